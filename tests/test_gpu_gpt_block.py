"""A GPT block in one call per direction (``ops.gpt_block``) against fp64 and against its layers one by one."""
import math

import pytest
import torch
import torch.utils.checkpoint

pytestmark = pytest.mark.gpu


@pytest.fixture
def calls(monkeypatch):
    from ghost_flow_b200 import ops

    seen, real = [], ops.gpt_block
    monkeypatch.setattr(ops, "gpt_block", lambda *a: seen.append(a) or real(*a))
    return seen


def _block(E, F, H, seed, bias=True, **kw):
    from ghost_flow_b200.models.configs import GPTConfig
    from ghost_flow_b200.models.gpt import GPTBlock

    m = GPTBlock(GPTConfig(n_embd=E, n_head=H, n_inner=F, dropout=0.0, **kw)).to(device="cuda", dtype=torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(seed)
    with torch.no_grad():
        for n, p in m.named_parameters():
            r = torch.randn(p.shape, generator=g, device="cuda")
            p.copy_(r / math.sqrt(p.shape[1]) if p.dim() == 2 else 1 + 0.1 * r if "ln" in n and "weight" in n else 0.1 * r)
    if not bias:
        for n in (m.attn.qkv, m.attn.out_proj, m.mlp.fc1, m.mlp.fc2, m.ln1, m.ln2):
            n.bias = None
    return m, g


def _want(m, x, dy):
    p = {n: t.detach().double().requires_grad_() for n, t in m.named_parameters()}
    x = x.detach().double().requires_grad_()
    B, S, E = x.shape
    H = m.attn.num_heads
    ln = lambda t, n: torch.nn.functional.layer_norm(t, (E,), p[n + ".weight"], p.get(n + ".bias"), 1e-5)  # noqa: E731
    lin = lambda t, n: torch.nn.functional.linear(t, p[n + ".weight"], p.get(n + ".bias"))  # noqa: E731
    q, k, v = (t.transpose(1, 2) for t in lin(ln(x, "ln1"), "attn.qkv").view(B, S, 3 * H, E // H).split(H, 2))
    s = q @ k.transpose(-1, -2) / math.sqrt(E // H)
    if m.attn.causal:
        s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=s.device).tril(), float("-inf"))
    h = x + lin((torch.softmax(s, -1) @ v).transpose(1, 2).reshape(B, S, E), "attn.out_proj")
    y = h + lin(torch.nn.functional.gelu(lin(ln(h, "ln2"), "mlp.fc1"), approximate="tanh"), "mlp.fc2")
    return y, dict(zip(["x", *p], torch.autograd.grad(y, [x, *p.values()], dy.double())))


def _pass(m, x, dy):
    m.zero_grad()
    x = x.detach().requires_grad_()
    y = m(x)
    y.backward(dy)
    return y.detach(), {"x": x.grad, **{n: p.grad for n, p in m.named_parameters()}}


# one and several query tiles, both head sizes, inner widths that are no whole tiles, products that split K (few rows, wide inner layer)
@pytest.mark.parametrize("B,S,E,F,H", [(1, 128, 128, 136, 2), (3, 256, 256, 1000, 2), (2, 384, 768, 3072, 12), (1, 128, 256, 4096, 4)])
@pytest.mark.parametrize("bias,causal", [(True, True), (False, False)])
def test_passes_match_fp64_and_the_layers(B, S, E, F, H, bias, causal, calls, kernel_status):
    m, g = _block(E, F, H, B + S, bias, causal=causal)
    x, dy = (torch.randn(B, S, E, generator=g, device="cuda").bfloat16() for _ in range(2))
    want, wgrad = _want(m, x, dy)
    y, grads = _pass(m, x, dy)
    assert len(calls) == 1
    hook = m.mlp.fc1.register_forward_hook(lambda *a: None)              # layer by layer
    y2, grads2 = _pass(m, x, dy)
    hook.remove()
    assert len(calls) == 1
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()  # noqa: E731
    for n in wgrad:
        # every tensor between two kernels is rounded to bf16 (2^-9) in both; the sums of a gradient with the one past the
        # branch once less in the one call
        e, e2 = rel(grads[n], wgrad[n]), rel(grads2[n], wgrad[n])
        assert e < 1.2e-2 and e < 1.05 * e2 + 2e-4, (n, e, e2)
    # the same launches; equal bits but where a product's slices of K are added in any order
    assert rel(y, want) < 8e-3 and rel(y, want) < 1.02 * rel(y2, want)
    if F < 2048:
        assert torch.equal(y, y2)


def test_frozen_parameters_no_gradient_and_accumulation(calls, kernel_status):
    m, g = _block(256, 512, 4, 1)
    x, dy = (torch.randn(2, 128, 256, generator=g, device="cuda").bfloat16() for _ in range(2))
    y, full = _pass(m, x, dy)
    with torch.no_grad():
        assert torch.equal(m(x), y)
    m.zero_grad()
    for n in (m.attn.qkv.weight, m.mlp.fc2.bias, m.ln1.weight):
        n.requires_grad_(False)
    xr = x.clone().requires_grad_()
    for _ in range(2):                                                   # twice: gradients add up
        m(xr).backward(dy)
    skip = {"attn.qkv.weight", "mlp.fc2.bias", "ln1.weight"}
    for n, p in m.named_parameters():
        assert (p.grad is None) == (n in skip)
        assert p.grad is None or torch.equal(p.grad, 2 * full[n])
    assert torch.equal(xr.grad, 2 * full["x"])
    m.requires_grad_(True)
    # a gradient that is no dense tensor, and saved tensors that a hook moves
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.cpu(), lambda t: t.cuda()):
        y2 = m(xr)
    m.zero_grad()
    y2.backward(dy.transpose(1, 2).contiguous().transpose(1, 2))
    assert torch.equal(y2, y)
    for n, p in m.named_parameters():
        assert torch.equal(p.grad, full[n]), n
    assert len(calls) == 5


def test_where_it_is_not_taken(calls):
    m, g = _block(256, 512, 4, 1)
    x = torch.randn(2, 128, 256, generator=g, device="cuda").bfloat16()
    m(x[:, :100])                                                        # a gradient, and no whole query tiles
    m(x.transpose(0, 1).contiguous().transpose(0, 1))
    m.mlp.drop.p = 0.1
    m(x)
    m.mlp.drop.p = 0.0
    m.attn.out_proj = torch.nn.Linear(256, 256).to(device="cuda", dtype=torch.bfloat16)
    m.attn.out_proj.forward = lambda t, residual: t + residual
    m(x)
    assert not calls
    m, _ = _block(256, 512, 4, 1)
    with torch.no_grad():
        assert m(x[:, :100].contiguous()).shape == (2, 100, 256) and len(calls) == 1
        m.float()(x.float())
    with torch.no_grad():
        m.cpu()(x.float().cpu())
    assert len(calls) == 1


@pytest.mark.parametrize("owner,name", [("", "ln1"), ("", "attn"), ("", "mlp"), ("attn", "qkv"), ("mlp", "fc2"), ("mlp", "act")])
def test_callables_in_the_place_of_modules_are_called(owner, name, calls):
    m, g = _block(256, 512, 4, 1)
    x = torch.randn(2, 128, 256, generator=g, device="cuda").bfloat16()
    want, o = m(x), m.get_submodule(owner)
    real = getattr(o, name)
    delattr(o, name)
    setattr(o, name, lambda *a, **k: real(*a, **k))
    assert torch.equal(m(x), want) and len(calls) == 1           # the layers' kernels on the same operands


@pytest.mark.parametrize("train,most", [(False, 1.02), (True, 1.25)])
def test_memory_of_a_pass_is_about_the_layers(train, most, calls):
    """Most memory held during a pass. Without a gradient nothing is kept for one; in the backward pass, which holds all results
    until its end where the layers let go of theirs one by one, temporaries share what they can (in rows of width 768, 2 bytes: 50
    against 42)."""
    m, g = _block(768, 3072, 12, 1)
    x, dy = (torch.randn(8, 1024, 768, generator=g, device="cuda").bfloat16() for _ in range(2))
    x.requires_grad_(train)

    def most_held():
        peak = 0
        for _ in range(2):                                               # the first one settles what is allocated once
            m.zero_grad()
            x.grad = None
            torch.cuda.synchronize()
            torch.cuda.reset_peak_memory_stats()
            before = torch.cuda.memory_allocated()
            with torch.set_grad_enabled(train):
                y = m(x)
            if train:
                y.backward(dy)
            torch.cuda.synchronize()
            peak = torch.cuda.max_memory_allocated() - before
            del y
        return peak

    one = most_held()
    assert len(calls) == 2
    hook = m.mlp.fc1.register_forward_hook(lambda *a: None)              # layer by layer
    layers = most_held()
    hook.remove()
    assert len(calls) == 2 and one <= most * layers, (one / 1e6, layers / 1e6)


def test_hooks_on_saved_tensors_get_typed_tensors(calls, kernel_status):
    """A hook that stores what it is given in another form goes by type and shape; bytes would be nothing to go by."""
    m, g = _block(256, 512, 4, 1)
    x, dy = (torch.randn(2, 128, 256, generator=g, device="cuda").bfloat16() for _ in range(2))
    y, full = _pass(m, x, dy)
    seen = []

    def through_the_host(t):
        seen.append((t.dtype, tuple(t.shape)))
        return t.t().contiguous().t().cpu() if t.dim() == 2 else t.double().cpu()

    with torch.autograd.graph.saved_tensors_hooks(lambda t: (t.dtype, through_the_host(t)), lambda p: p[1].cuda().to(p[0])):
        y2, grads = _pass(m, x, dy)
    assert len(calls) == 2 and torch.equal(y, y2)
    for n in full:
        assert torch.equal(grads[n], full[n]), n
    bf16, fp32 = torch.bfloat16, torch.float32
    assert {t for t, _ in seen} == {bf16, fp32}
    for want in ((bf16, (2, 128, 256)), (bf16, (2, 128, 512)), (bf16, (2, 128, 12, 64)), (fp32, (2, 4, 128)), (fp32, (2, 256))):
        assert want in seen
    y3 = torch.utils.checkpoint.checkpoint(m, x.clone().requires_grad_(), use_reentrant=False)
    m.zero_grad()
    y3.backward(dy)
    for n, p in m.named_parameters():
        assert torch.equal(p.grad, full[n]), n
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t, lambda t: t.float() if t.shape == (2, 128, 512) else t):
        y4 = m(x.clone().requires_grad_())
    with pytest.raises(RuntimeError, match="a hook returned a saved tensor"):
        y4.backward(dy)


def test_a_ragged_sequence_with_a_gradient_is_not_taken(calls):
    """Dense operands: it is the sequence, which the backward kernels do not have, that the layers are asked about."""
    m, g = _block(256, 512, 4, 1)
    x = torch.randn(2, 100, 256, generator=g, device="cuda").bfloat16()
    assert x.is_contiguous()
    y = m(x)
    assert not calls and y.requires_grad
    with pytest.raises(RuntimeError, match="multiple of 128"):
        y.backward(torch.ones_like(y))
    m.requires_grad_(False)
    m(x)
    assert len(calls) == 1                                               # nothing to differentiate: taken


# one token, rows that go to the few-row kernels (alone and as a batch), lengths around a query tile, sequences that end inside one
@pytest.mark.parametrize("B,S", [(1, 1), (1, 17), (3, 20), (1, 64), (2, 100), (1, 129), (5, 127), (1, 300)])
@pytest.mark.parametrize("E,F,H,causal", [(256, 512, 4, True), (768, 3072, 12, False), (256, 4096, 2, True)])
def test_any_length_without_a_gradient(B, S, E, F, H, causal, calls, kernel_status):
    m, g = _block(E, F, H, S, causal=causal)
    x = torch.randn(B, S, E, generator=g, device="cuda").bfloat16()
    want, _ = _want(m, x, torch.ones_like(x))
    with torch.no_grad():
        y = m(x)
        assert len(calls) == 1
        hook = m.mlp.fc1.register_forward_hook(lambda *a: None)          # layer by layer
        y2 = m(x)
        hook.remove()
        assert len(calls) == 1
    rel = lambda a, b: ((a.double() - b).norm() / b.norm()).item()  # noqa: E731
    assert rel(y, want) < 8e-3 and rel(y, want) < 1.02 * rel(y2, want)   # as above
    if F < 2048:
        assert torch.equal(y, y2)
