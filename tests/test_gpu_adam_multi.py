"""Adam / AdamW over many tensors in one launch (``gf_adam_multi``) against the update in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _reference(p, g, m, v, step, lr, wd, decoupled):
    p, g = p.double(), g.double()
    if not decoupled:
        g = g + wd * p
    m.mul_(0.9).add_(g, alpha=0.1)
    v.mul_(0.999).addcmul_(g, g, value=0.001)
    if decoupled:
        p = p * (1 - lr * wd)
    return p - lr * (m / (1 - 0.9 ** step)) / ((v / (1 - 0.999 ** step)).sqrt() + 1e-8)


# sizes around a vector of four, a thread block's share (4096) and the table's length (100 rows to a launch)
@pytest.mark.parametrize("sizes", [[1], [3, 4, 5], [4095, 4096, 4097, 12289], [7] * 203, [1 << 20]])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("decoupled", [True, False])
def test_update_matches_64_bits(sizes, dtype, decoupled):
    from ghost_flow_b200.ops import _lib
    from ghost_flow_b200.optim import Adam, AdamW

    gen = torch.Generator(device="cuda").manual_seed(sum(sizes))
    ps = [torch.nn.Parameter(torch.randn(n, generator=gen, device="cuda").to(dtype)) for n in sizes]
    ref = [p.detach().double() for p in ps]
    ms, vs = [torch.zeros_like(r) for r in ref], [torch.zeros_like(r) for r in ref]
    opt = (AdamW if decoupled else Adam)(ps, lr=1e-2, weight_decay=0.1)
    for step in (1, 2, 3):
        for i, p in enumerate(ps):
            g = torch.randn(p.numel() + 1, generator=gen, device="cuda").to(dtype)
            # every third gradient is a view that starts on no vector boundary, every fifth is missing in step 2
            g = g[1:] if i % 3 == 2 else g[:-1].clone()
            p.grad = None if (i % 5 == 4 and step == 2) else g
            if p.grad is not None:
                ref[i] = _reference(ref[i], g, ms[i], vs[i], step, 1e-2, 0.1, decoupled)
        n0 = _lib.launch_count()
        opt.step()
        assert _lib.launch_count() - n0 <= (len(ps) + 99) // 100
    for p, r in zip(ps, ref):
        # fp32: about ten roundings of 2^-24 a step, and 1 - beta2 as a float is off by 2^-15 of itself (v, so the update by half)
        if dtype == torch.float32:
            assert torch.allclose(p.detach().double(), r, rtol=2e-6, atol=2e-6)
        else:
            assert torch.allclose(p.detach().double(), r, rtol=2 ** -8, atol=2e-6)


def test_layouts_that_need_the_flat_copy_give_the_same_result():
    from ghost_flow_b200.optim import AdamW

    gen = torch.Generator(device="cuda").manual_seed(0)
    w = torch.randn(48, 40, generator=gen, device="cuda", dtype=torch.bfloat16)
    g = torch.randn(40, 48, generator=gen, device="cuda", dtype=torch.bfloat16)
    a, b = torch.nn.Parameter(w.clone()), torch.nn.Parameter(w.clone())
    oa, ob = AdamW([a]), AdamW([b])
    for _ in range(2):
        a.grad, b.grad = g.t(), g.t().contiguous()      # strided gradient: gathered; contiguous: read in place
        oa.step()
        ob.step()
    assert torch.equal(a, b)


def test_empty_parameters_and_shared_storage():
    from ghost_flow_b200.optim import AdamW

    w = torch.randn(64, device="cuda").bfloat16()
    tied = [torch.nn.Parameter(w.clone()) for _ in range(2)]
    tied[1].data = tied[0].data
    alone = torch.nn.Parameter(w.clone())
    empty = torch.nn.Parameter(torch.zeros(0, 3, device="cuda"))
    for p in (*tied, alone, empty):
        p.grad = torch.ones_like(p)
    tied[0].grad.neg_()
    AdamW([*tied, empty], lr=0.1).step()
    AdamW([empty, alone], lr=0.1).step()
    assert torch.equal(tied[0], alone)          # the second of the two parameters is written last
    AdamW([empty], lr=0.1).step()


def test_overlapping_weights_are_copied_back_in_order():
    from ghost_flow_b200.optim import AdamW

    w = torch.randn(96, device="cuda").bfloat16()
    buf, alone = w.clone(), [torch.nn.Parameter(w[lo:lo + 64].clone()) for lo in (0, 32)]
    ps = [torch.nn.Parameter(buf[lo:lo + 64]) for lo in (0, 32)]
    for p, q in zip(ps, alone):
        q.grad = torch.randn(64, device="cuda").bfloat16()
        p.grad = q.grad.clone()
    AdamW(ps, lr=0.1).step()
    AdamW(alone, lr=0.1).step()
    assert torch.equal(buf, torch.cat((alone[0].detach()[:32], alone[1].detach())))    # the second is written last


def test_loaded_master_weights_reach_parameters_without_a_gradient():
    from ghost_flow_b200.optim import AdamW

    def make():
        g = torch.Generator(device="cuda").manual_seed(3)
        ps = [torch.nn.Parameter(torch.randn(40, generator=g, device="cuda").bfloat16()) for _ in range(3)]
        return ps, AdamW(ps, lr=0.1)

    ps, opt = make()
    for p in ps:
        p.grad = torch.ones_like(p)
    opt.step()
    saved, want = opt.state_dict(), [p.detach().clone() for p in ps]
    qs, other = make()
    other.load_state_dict(saved)                    # the optimizer alone: its master copies are the truth
    qs[0].grad = torch.zeros_like(qs[0])
    other.step()
    assert torch.equal(qs[1], want[1]) and torch.equal(qs[2], want[2])
