"""Products whose K is split over CTA pairs (``gemm2sm_run_sliced``) against fp64: ragged tiles and parts, all layouts, what is added."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# 16 tiles of 256 x 256 at least; two to four parts of K, of unequal numbers of 64-wide blocks and with a rest
@pytest.mark.parametrize("M,N,K,parts", [(1024, 1024, 2048, 4), (1000, 1000, 2120, 4), (2304, 768, 8192, 2), (1288, 1272, 4104, 2),
                                         (256, 4096, 4096, 4), (1600, 1600, 8192, 3)])
@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, False), (True, True)])
def test_parts_of_k_add_up(M, N, K, parts, a_mn, b_mn, kernel_status):
    from ghost_flow_b200.ops.gemm import _workspace, gemm_raw

    assert _workspace(M, N, K, a_mn, b_mn, True, False, False) == parts * M * N
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn(M, K, generator=g, device="cuda").bfloat16()
    b = torch.randn(N, K, generator=g, device="cuda").bfloat16()
    bias = torch.randn(N, generator=g, device="cuda").bfloat16()
    res = torch.randn(M, N + 3, generator=g, device="cuda").bfloat16()[:, :N]          # rows off 8-byte boundaries
    sa, sb = a.t().contiguous() if a_mn else a, b.t().contiguous() if b_mn else b
    prod = a.double() @ b.double().t()
    # fp32 sums of K products of size one, of which each of K / 16 steps may lose 2^-23, and one rounding to bf16
    tol = dict(rtol=2 ** -8, atol=K * 2 ** -20)
    y = gemm_raw(sa, a_mn, sb, b_mn, M, N, K)
    assert torch.allclose(y.double(), prod, **tol)
    assert torch.equal(y, gemm_raw(sa, a_mn, sb, b_mn, M, N, K))                       # the order of the sums is fixed
    wide = torch.full((M, N + 1), 7.0, device="cuda", dtype=torch.bfloat16)
    gemm_raw(sa, a_mn, sb, b_mn, M, N, K, out=wide[:, :N], bias=bias, residual=res, alpha=0.5)
    assert torch.allclose(wide[:, :N].double(), 0.5 * prod + bias.double() + res.double(), **tol) and (wide[:, N] == 7).all()


def test_what_is_not_split_here():
    from ghost_flow_b200.ops.gemm import _workspace

    for M, N, K in [(1024, 1024, 2040), (255, 8192, 4096), (768, 768, 8192), (4096, 4096, 4096)]:
        assert _workspace(M, N, K, True, True, True, False, False) <= M * N
    assert _workspace(1024, 1024, 4096, True, True, True, True, False) == 0            # adds to what is there
    assert _workspace(1024, 1024, 4096, True, True, True, False, True) == 0            # an activation
