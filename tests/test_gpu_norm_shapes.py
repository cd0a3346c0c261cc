"""Norms and column sums at the edges of their kernels (one warp / one CTA per row, vectors per thread, rows per grid) against
fp64, forward and backward."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# row lengths around one warp's and one CTA's steps; row counts below, at and beyond a grid of rows
SHAPES = [(1, 8), (3, 256), (9, 264), (17, 768), (8, 1016), (5, 1024), (5, 1032), (700, 2048), (3, 2056), (1500, 4096),
          (2, 4104), (601, 8192), (5000, 128),
          # rows of 264 to 1024 columns: one to a CTA while there are few of them (740 forward, 148 backward), else one to a warp
          (148, 264), (149, 264), (740, 768), (741, 768), (900, 1016), (1400, 1024)]


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm().clamp_min(1e-30)).item()


@pytest.mark.parametrize("T,D", SHAPES)
@pytest.mark.parametrize("kind", ["rms", "rms_res", "ln", "ln_nobias"])
def test_norms_match_fp64(T, D, kind):
    from ghost_flow_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T + D)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, w, b, r, dy, dh = mk(T, D).requires_grad_(), mk(D).requires_grad_(), mk(D).requires_grad_(), mk(T, D).requires_grad_(), mk(T, D), mk(T, D)
    h64 = (x + r).detach().double().requires_grad_() if kind == "rms_res" else x.detach().double().requires_grad_()
    w64, b64 = w.detach().double().requires_grad_(), b.detach().double().requires_grad_()
    if kind.startswith("rms"):
        want = h64 * torch.rsqrt(h64.square().mean(-1, keepdim=True) + 1e-6) * w64
        if kind == "rms_res":
            y, h = ops.rms_norm(x, w, 1e-6, residual=r)
            assert torch.equal(h, (x + r).detach())
            torch.autograd.backward([y, h], [dy, dh])
        else:
            y = ops.rms_norm(x, w, 1e-6)
            y.backward(dy)
    else:
        bias = b if kind == "ln" else None
        want = torch.nn.functional.layer_norm(h64, (D,), w64, b64 if kind == "ln" else None, 1e-5)
        y = ops.layer_norm(x, w, bias, 1e-5)
        y.backward(dy)
    want.backward(dy.double())
    dx = h64.grad + (dh.double() if kind == "rms_res" else 0)
    # one bf16 store of an fp32 result: 2^-9 at most, 0.0017 over a whole tensor; a row of eight may cancel to a tenth of it
    assert _rel(y, want.detach()) < 4e-3
    assert _rel(x.grad, dx) < (2e-2 if D == 8 else 4e-3)
    assert _rel(w.grad, w64.grad) < 4e-3
    if kind == "rms_res":
        assert torch.equal(r.grad, x.grad)
    if kind == "ln":
        assert _rel(b.grad, b64.grad) < 4e-3
    with torch.no_grad():                    # without row statistics
        z = ops.rms_norm(x, w, 1e-6) if kind == "rms" else ops.rms_norm(x, w, 1e-6, residual=r)[0] if kind == "rms_res" \
            else ops.layer_norm(x, w, b if kind == "ln" else None, 1e-5)
    assert torch.equal(z, y)


@pytest.mark.parametrize("T,D", SHAPES + [(8, 256), (33, 2304), (4099, 3072)])
def test_column_sums_match_fp64(T, D):
    from ghost_flow_b200.ops.gemm import _colsum

    x = torch.randn(T, D + 8, device="cuda").bfloat16()[:, :D]
    s = x.double().sum(0)
    # fp32 sums of T values and one bf16 rounding
    assert torch.allclose(_colsum(x).double(), s, rtol=2 ** -8, atol=T * 2 ** -22)


@pytest.mark.parametrize("ln", [False, True])
def test_scratch_of_a_recorded_backward_pass_stays_its_own(ln):
    from ghost_flow_b200 import ops

    def step(x, w, dy):
        y = ops.layer_norm(x, w, None) if ln else ops.rms_norm(x, w)
        return torch.autograd.grad(y, (x, w), dy)

    def data(T, D):
        return (torch.randn(T, D, device="cuda").bfloat16().requires_grad_(), torch.ones(D, device="cuda").bfloat16().requires_grad_(),
                torch.randn(T, D, device="cuda").bfloat16())

    small, large = data(300, 256), data(4000, 8192)
    want = [g.clone() for g in step(*small)]
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        step(*small)
    torch.cuda.current_stream().wait_stream(s)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step(*small)
    first = [g.clone() for g in step(*large)]
    # everything that the larger call gave back is taken by tensors of the program, which a replay must leave alone
    held = [torch.zeros(1 << 20, device="cuda") for _ in range(64)]
    graph.replay()
    for g, w in zip(got, want):
        assert torch.equal(g, w)
    assert not any(t.any() for t in held)

    # two streams in flight: each call has its own partial sums
    streams, out = [torch.cuda.Stream() for _ in range(2)], [[], []]
    torch.cuda.synchronize()
    for _ in range(8):
        for i, (s, d) in enumerate(zip(streams, (small, large))):
            with torch.cuda.stream(s):
                out[i].append(step(*d))
    torch.cuda.synchronize()
    for i, w in enumerate((want, first)):
        for gs in out[i]:
            assert all(torch.equal(a, b) for a, b in zip(gs, w))
