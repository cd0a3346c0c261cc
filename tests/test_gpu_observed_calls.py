"""The paths that compute several modules in one call (GPT block, LLaMA decoder layer, norm in the head) under what follows the calls of
modules and operations: not taken, and the outcome is the layers'."""
import math

import pytest
import torch
import torch.autograd.forward_ad as fwd_ad
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

pytestmark = pytest.mark.gpu


class _Dispatch(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class _Function(TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


@pytest.fixture
def taken(monkeypatch):
    from ghost_flow_b200 import ops
    from ghost_flow_b200.ops import raw

    seen = []
    for where, name in ((ops, "gpt_block"), (raw, "llama_decode_layer"), (raw, "rmsnorm_gemm")):
        real = getattr(where, name)
        monkeypatch.setattr(where, name, lambda *a, real=real, name=name: seen.append(name) or real(*a))
    return seen


def _random(m, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    with torch.no_grad():
        for p in m.parameters():
            r = torch.randn(p.shape, generator=g, device="cuda")
            p.copy_(r / math.sqrt(p.shape[1]) if p.dim() == 2 else 1 + 0.1 * r)
    return m, g


def _gpt():
    from ghost_flow_b200.models.configs import GPTConfig
    from ghost_flow_b200.models.gpt import GPTBlock

    m, g = _random(GPTBlock(GPTConfig(n_embd=256, n_head=4, n_inner=512, dropout=0.0)).to(device="cuda", dtype=torch.bfloat16), 1)
    return m, m, torch.randn(2, 128, 256, generator=g, device="cuda").bfloat16()


def _llama(what):
    """The layer (``x``) or the model (``ids``): each call decodes position 7 on caches of the same content."""
    from ghost_flow_b200 import ops
    from ghost_flow_b200.models import LLaMAConfig, LLaMAForCausalLM
    from ghost_flow_b200.models.llama import LLaMADecoderLayer

    cfg = LLaMAConfig(vocab_size=512, hidden_size=256, intermediate_size=512, num_hidden_layers=1, num_attention_heads=4,
                      num_key_value_heads=2, max_position_embeddings=128)
    m, g = _random((LLaMADecoderLayer if what == "layer" else LLaMAForCausalLM)(cfg, device="cuda", dtype=torch.bfloat16), 2)
    cos, sin = ops.rope_tables(128, 64, 10000.0, "cuda")
    old = [torch.randn(2, 40, 2, 64, generator=g, device="cuda").bfloat16() for _ in range(2)]
    if what == "layer":
        f = lambda x: m(x, cos, sin, cache=tuple(c.clone() for c in old), start_pos=7)  # noqa: E731
        return m, f, torch.randn(2, 1, 256, generator=g, device="cuda").bfloat16()
    f = lambda ids: m(ids, caches=[tuple(c.clone() for c in old)], start_pos=7)  # noqa: E731
    return m, f, torch.randint(0, 512, (2, 1), generator=g, device="cuda")


def _case(what):
    return _gpt() if what == "gpt" else _llama(what)


@pytest.mark.parametrize("what", ["gpt", "layer", "model"])
def test_modes_and_subclasses_run_layer_by_layer(what, taken, kernel_status):
    m, f, a = _case(what)
    with torch.no_grad():
        f(a)
        n = len(taken)
        assert n
        hooks = [t.register_forward_hook(lambda *a: None) for t in m.modules()]      # every module is called
        want = f(a)
        for h in hooks:
            h.remove()
        with _Dispatch():
            assert torch.equal(f(a), want)
        with _Function():
            assert torch.equal(f(a), want)
        with fwd_ad.dual_level():
            assert torch.equal(f(a), want)
            if what != "model":
                assert torch.equal(fwd_ad.unpack_dual(f(fwd_ad.make_dual(a, torch.ones_like(a)))).primal, want)
        if what != "model":
            assert torch.equal(f(a.as_subclass(type("Sub", (torch.Tensor,), {}))).as_subclass(torch.Tensor), want)
    assert len(taken) == n


def test_traced_block_runs_layer_by_layer(taken):
    """Launches escape a trace, the layers' as well: what counts is that nothing more does."""
    m, _, x = _gpt()
    m.requires_grad_(False)
    torch.jit.trace(m, (x,), check_trace=False)
    assert not taken


@pytest.mark.parametrize("transform", [
    lambda f, a: torch.func.vmap(f)(torch.stack((a, a))), lambda f, a: torch.func.jvp(f, (a,), (torch.ones_like(a),)),
    lambda f, a: torch.func.grad(lambda t: f(t).float().sum())(a)])
@pytest.mark.parametrize("what", ["gpt", "layer"])
def test_transforms_are_refused_by_the_layers(what, transform, taken):
    """By autograd, which says what it misses, and not by a tensor without memory."""
    _, f, a = _case(what)
    if what == "layer" and transform.__code__.co_names[-1:] == ("stack",):
        pytest.skip("caches are not batched")
    with pytest.raises(RuntimeError, match="autograd.Function with functorch transforms"):
        transform(f, a)
    assert not taken


@pytest.mark.parametrize("what", ["gpt", "layer", "model"])
def test_transforms_without_gradients_never_meet_the_call(what, taken):
    _, f, a = _case(what)
    with torch.no_grad(), pytest.raises(RuntimeError):
        torch.func.vmap(f, randomness="same")(torch.stack((a, a)))
    assert not taken


@pytest.mark.parametrize("what", ["gpt", "layer", "model"])
def test_device_contexts_change_nothing(what, taken, kernel_status):
    _, f, a = _case(what)
    with torch.no_grad():
        want = f(a)
        n = len(taken)
        for device in ("cuda", "cpu", "meta"):            # every allocation next to a launch names its device
            with torch.device(device):
                assert torch.equal(f(a), want)
        assert len(taken) == 4 * n
