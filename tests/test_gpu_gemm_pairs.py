"""CTA-pair GEMM: products with nothing to add (four epilogue warps) against the same with a bias of zeros (eight), and fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# 74 tiles of 256 x 256 and more, ragged in rows and columns; narrow outputs take tiles of 256 x 128
@pytest.mark.parametrize("M,N,K", [(4096, 2048, 256), (2050, 2312, 264), (19000, 72, 512), (304, 9600, 328)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_plain_products_equal_those_with_a_zero_bias(M, N, K, a_mn, b_mn, dtype, kernel_status):
    from ghost_flow_b200.ops.gemm import gemm_raw

    M, N = (M + 7) // 8 * 8, (N + 7) // 8 * 8
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    b = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    sa, sb = a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b
    plain = gemm_raw(sa, a_mn, sb, b_mn, M, N, K, out_dtype=dtype, alpha=0.5)
    assert torch.equal(plain, gemm_raw(sa, a_mn, sb, b_mn, M, N, K, out_dtype=dtype, alpha=0.5,
                                       bias=torch.zeros(N, device="cuda", dtype=torch.bfloat16)))
    want = 0.5 * (a.double() @ b.double().t())
    # sums of K products of size one, of which each of K / 16 steps may lose 2^-23, and one rounding to bf16
    assert torch.allclose(plain.double(), want, rtol=2 ** -8 if dtype == torch.bfloat16 else 1e-5, atol=K * 2 ** -20)
