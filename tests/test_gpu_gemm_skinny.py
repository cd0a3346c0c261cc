"""GEMM of at most 16 rows (``gemm_skinny.cu``) against fp64, at the edges of its tiles and of the rule that picks it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# 8 / 16 rows to a tile, 16 features to a block, 64-wide k blocks (two to a warp and round, eight warps): 1024 to a round
@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17])
@pytest.mark.parametrize("N,K", [(8, 8), (16, 64), (24, 72), (1000, 1016), (520, 1024), (17, 1032), (1, 2048), (4096, 4104),
                                 (24, 4096), (24, 4104), (2056, 4112), (40, 6144), (40, 6152), (1544, 6176), (264, 8200)])
def test_skinny_gemm_matches_fp64(M, N, K):
    from ghost_flow_b200.ops.gemm import gemm_raw

    g = torch.Generator(device="cuda").manual_seed(M * 7919 + N * 31 + K)
    a = torch.randn(M, K + 8, generator=g, device="cuda").bfloat16()[:, :K]           # pitch beyond the row
    w = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    bias = torch.randn(N, generator=g, device="cuda").bfloat16()
    res = torch.randn(M, (N + 15) // 8 * 8, generator=g, device="cuda").bfloat16()[:, :N]
    prod = a.double() @ w.double().t()
    # fp32 sums of K products of size one: rounding errors of about sqrt(K) * 2^-24 * sqrt(K), and one bf16 rounding
    tol = dict(rtol=2 ** -8, atol=K * 2 ** -22)
    y = gemm_raw(a, False, w, False, M, N, K)
    assert y.shape == (M, N) and torch.allclose(y.double(), prod, **tol)
    y = gemm_raw(a, False, w, False, M, N, K, bias=bias, residual=res, alpha=0.5)
    assert torch.allclose(y.double(), 0.5 * prod + bias.double() + res.double(), **tol)
    y = gemm_raw(a, False, w, False, M, N, K, bias=bias, relu=True)
    assert torch.allclose(y.double(), (prod + bias.double()).clamp(min=0), **tol)
    y = gemm_raw(a, False, w, False, M, N, K, out_dtype=torch.float32)
    assert y.dtype == torch.float32 and torch.allclose(y.double(), prod, rtol=1e-5, atol=K * 2 ** -22)


def test_forms_that_keep_the_general_path():
    from ghost_flow_b200.ops.gemm import gemm_raw

    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn(8, 64, generator=g, device="cuda").bfloat16()
    w = torch.randn(48, 64, generator=g, device="cuda").bfloat16()
    want = a.double() @ w.double().t()
    tol = dict(rtol=2 ** -8, atol=2 ** -16)
    assert torch.allclose(gemm_raw(a, False, w.t().contiguous(), True, 8, 48, 64).double(), want, **tol)
    assert torch.allclose(gemm_raw(a.t().contiguous(), True, w, False, 8, 48, 64).double(), want, **tol)
    assert torch.allclose(gemm_raw(a, False, w, False, 8, 48, 64, bn_hint=128).double(), want, **tol)
    out = torch.ones(8, 48, device="cuda", dtype=torch.float32)
    gemm_raw(a, False, w, False, 8, 48, 64, out=out, accumulate=True)
    assert torch.allclose(out.double(), want + 1, rtol=1e-5, atol=2 ** -16)
    # a contraction that is no whole number of 16-byte vectors (the pitch is)
    short = gemm_raw(a[:, :60], False, w[:, :60], False, 8, 48, 60)
    assert torch.allclose(short.double(), a[:, :60].double() @ w[:, :60].double().t(), **tol)
