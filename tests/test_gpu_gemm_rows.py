"""Few-row GEMM (``gemm_rows.cu``) against fp64 at the edges of its token tiles, feature tiles, ring and clusters, with its inputs."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(x, w, out, M, N, K, inp, norm_w, bias, res, alpha, relu):
    import ctypes

    from ghost_flow_b200.ops import _lib

    lib = _lib.cuda_lib()
    P, L, I, F = ctypes.c_void_p, ctypes.c_longlong, ctypes.c_int, ctypes.c_float
    lib.gf_gemm_rows.argtypes = [P, L, P, L, P, L, I, I, I, I, I, P, F, P, P, L, F, I, P, P]
    p = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    rc = lib.gf_gemm_rows(p(x), x.stride(0), p(w), w.stride(0), p(out), out.stride(0), out.dtype == torch.float32, M, N, K, inp,
                          p(norm_w), 1e-5, p(bias), p(res), res.stride(0) if res is not None else 0, alpha, relu,
                          _lib.status_word(x.device).data_ptr(), _lib.stream_ptr())
    _lib.check_status()
    return rc


# 16 / 32 / 64 tokens and 128 features to a tile, blocks of 64 of K, four to each CTA of a cluster of 1, 2, 4 or 8, a ring of 4 to 6
@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(1, 8), (127, 72), (129, 256), (130, 504), (1000, 520), (256, 1032), (40, 2056), (4096, 4104), (38000, 64)])
def test_against_fp64(M, N, K):
    g = torch.Generator(device="cuda").manual_seed(M * 7919 + N * 31 + K)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    w, norm_w, bias, res = mk(N, K), 1 + 0.1 * mk(K), mk(N), mk(M, N + 3)[:, :N]
    for inp in (0, 1, 2) if M <= 16 else (0,):
        x = mk(M, K * (2 if inp == 2 else 1) + 8)[:, :K * (2 if inp == 2 else 1)]         # pitch beyond the row
        xd = x.double()
        if inp == 1:
            xd = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5) * norm_w.double()
        if inp == 2:
            xd = torch.nn.functional.silu(xd[:, :K]) * xd[:, K:]
        prod = xd @ w.double().t()
        # fp32 sums of K products: about K * 2^-24 of their size, 2^-22 with room; an input that is computed is rounded to bf16
        # first, 2^-9 of each term, which add up like their square root
        size = (xd.square() @ w.double().t().square()).sqrt()
        tol = K * 2 ** -22 + (6 * 2 ** -9 * size if inp else 0)
        for dtype, rnd in ((torch.float32, 2 ** -20), (torch.bfloat16, 2 ** -8)):
            out = torch.full((M, N + 5), 7.0, device="cuda", dtype=dtype)
            assert _run(x, w, out[:, :N], M, N, K, inp, norm_w, None, None, 1.0, 0) == 0
            assert ((out[:, :N].double() - prod).abs() <= tol + rnd * prod.abs()).all() and (out[:, N:] == 7).all()
        out = torch.empty((M, N), device="cuda", dtype=torch.bfloat16)
        for r in (res, res.contiguous()):                          # rows off and on boundaries of four values
            assert _run(x, w, out, M, N, K, inp, norm_w, bias, r, 0.5, 1) == 0
            want = (0.5 * prod + bias.double() + r.double()).clamp(min=0)
            assert ((out.double() - want).abs() <= tol + 2 ** -8 * want).all()


def test_what_is_refused():
    t = torch.zeros(128, 128, device="cuda", dtype=torch.bfloat16)
    assert _run(t, t, t, 65, 8, 64, 0, None, None, None, 1.0, 0) != 0            # more rows than the tile has
    assert _run(t, t, t, 17, 8, 64, 1, t, None, None, 1.0, 0) != 0               # a computed input of more than 16
    assert _run(t, t, t, 8, 8, 60, 0, None, None, None, 1.0, 0) != 0             # no whole 16-byte vectors


def test_nothing_finite_hides_what_is_not():
    """An infinite or NaN token spoils its own row only."""
    x = torch.ones(8, 256, device="cuda", dtype=torch.bfloat16)
    x[2, 7], x[5, 200] = float("inf"), float("nan")
    w = torch.full((200, 256), 0.5, device="cuda", dtype=torch.bfloat16)
    norm_w = torch.ones(256, device="cuda", dtype=torch.bfloat16)
    for inp in (0, 1):
        out = torch.empty(8, 200, device="cuda", dtype=torch.bfloat16)
        assert _run(x, w, out, 8, 200, 256, inp, norm_w, None, None, 1.0, 0) == 0
        bad = ~torch.isfinite(out).all(1)
        assert bad.tolist() == [i in (2, 5) for i in range(8)] and torch.isnan(out[5]).all()


@pytest.mark.parametrize("M,ctas", [(16, 3), (32, 2), (64, 2)])
def test_all_clusters_of_a_product_fit_on_the_machine(M, ctas, kernel_status):
    """Clusters lie within GPCs, so fewer of them fit than SMs and CTAs to an SM say: one that does not fit is a second wave."""
    from ghost_flow_b200.ops import _lib

    ask = _lib.cuda_lib().gf_gemm_rows_clusters
    slots = ctas * torch.cuda.get_device_properties(0).multi_processor_count
    fit = {s: ask(M, 1, 1, s) for s in (1, 2, 4, 8)}
    assert all(0 < fit[s] <= slots // s for s in fit) and fit[8] <= fit[4] <= fit[2] <= fit[1] == slots
    for K in (64, 512, 1024, 2048, 4096):
        # around the numbers of tiles where a cluster size stops to fit, by machine and by slots
        for tiles in {t + d for s in (2, 4, 8) for t in (fit[s], slots // s) for d in (0, 1)} | {1}:
            most = max(s for s in (1, 2, 4, 8) if s == 1 or (tiles <= fit[s] and 4 * s <= K // 64))
            assert ask(M, 128 * tiles, K, 0) == ask(M, 128 * tiles - 127, K, 0) == most, (K, tiles)
    g = torch.Generator(device="cuda").manual_seed(M)
    for tiles in (fit[8] + 1, fit[4] + 1, fit[2] + 1):
        x, w = (torch.randn(n, 2048, generator=g, device="cuda").bfloat16() for n in (M, 128 * tiles))
        out = torch.empty(M, 128 * tiles, device="cuda", dtype=torch.bfloat16)
        assert _run(x, w, out, M, 128 * tiles, 2048, 0, None, None, None, 1.0, 0) == 0
        want = x.double() @ w.double().t()
        # fp32 sums of 2048 products, about 2048 * 2^-22 with room, and the rounding of the result
        assert ((out.double() - want).abs() <= 2048 * 2 ** -22 + 2 ** -8 * want.abs()).all()


def test_tiles_that_never_fit_at_once(kernel_status):
    """More tiles than the machine holds whole: a long K is cut in two where the last ones are few."""
    from ghost_flow_b200.ops import _lib

    ask = _lib.cuda_lib().gf_gemm_rows_clusters
    for M in (16, 32, 64):
        whole = ask(M, 1, 1, 1)
        for K, tiles, want in ((4096, whole + 1, 2), (4096, whole + whole // 4, 2), (4032, whole + 1, 1), (4096, 2 * whole, 2 if M == 16 else 1),
                               (8192, whole, 1)):
            assert ask(M, 128 * tiles, K, 0) == want, (M, K, tiles)
    g = torch.Generator(device="cuda").manual_seed(1)
    M, N, K = 16, 128 * (ask(16, 1, 1, 1) + 3) - 5, 4096
    x, w, norm_w = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((M, K), (N, K), (K,)))
    out = torch.empty(M, N + 5, device="cuda", dtype=torch.bfloat16)[:, :N]
    for inp in (0, 1):
        assert _run(x, w, out, M, N, K, inp, norm_w, None, None, 1.0, 0) == 0
        xd = x.double()
        if inp:
            xd = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5) * norm_w.double()
        want = xd @ w.double().t()
        size = (xd.square() @ w.double().t().square()).sqrt()                # tolerances as above
        assert ((out.double() - want).abs() <= K * 2 ** -22 + (6 * 2 ** -9 * size if inp else 0) + 2 ** -8 * want.abs()).all()
