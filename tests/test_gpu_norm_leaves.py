"""RMSNorm with a residual: two leaves get gradients of their own, equal ones, whatever else the graph does with them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,D", [(1, 128), (700, 1024), (40, 4096), (9, 8192)])
def test_gradients_of_two_leaves(T, D):
    from ghost_flow_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(T)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, r, w, dy, dh = mk(T, D), mk(T, D), mk(D), mk(T, D), mk(T, D)

    def grads(a, b):
        leaves = [t for t in (a, b, wl) if t.requires_grad and t.is_leaf]
        y, h = ops.rms_norm(a, wl, 1e-6, residual=b)
        return torch.autograd.grad([y, h], leaves, [dy, dh])

    wl = w.clone().requires_grad_()
    xl, rl = x.clone().requires_grad_(), r.clone().requires_grad_()
    gx, gr, gw = grads(xl, rl)
    assert gx.data_ptr() != gr.data_ptr() and torch.equal(gx, gr)
    # one of them frozen, or no leaf: one gradient, the same numbers
    assert torch.equal(grads(xl, r)[0], gx) and torch.equal(grads(x, rl)[0], gx)
    y, h = ops.rms_norm(xl * 1, wl, 1e-6, residual=rl)
    a, b = torch.autograd.grad([y, h], [xl, rl], [dy, dh])
    assert torch.equal(a, gx) and torch.equal(b, gx)
    # the same leaf on both sides: the sum
    y, h = ops.rms_norm(xl, wl, 1e-6, residual=xl)
    (s,) = torch.autograd.grad([y, h], [xl], [dy, dh])
    y, h = ops.rms_norm(xl * 1, wl, 1e-6, residual=xl * 1)
    (s2,) = torch.autograd.grad([y, h], [xl], [dy, dh])
    assert torch.equal(s, s2)
