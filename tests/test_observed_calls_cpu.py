"""When a call may be replaced by a kernel launch that tensor-level tools do not see."""
import torch
from torch.autograd import forward_ad
from torch.utils._python_dispatch import TorchDispatchMode

from ghost_flow_b200.ops import fused


class _Mode(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def test_every_observer_is_noticed():
    assert not fused._observed()
    seen = []
    with _Mode():
        seen.append(fused._observed())
    with forward_ad.dual_level():
        seen.append(fused._observed())
    with torch.overrides.TorchFunctionMode():
        seen.append(fused._observed())
    torch.vmap(lambda x: seen.append(fused._observed()) or x)(torch.ones(2))
    torch.jit.trace(lambda x: seen.append(fused._observed()) or x + 1, torch.ones(2), check_trace=False)
    assert seen == [True] * 5 and not fused._observed()


def test_a_torch_without_one_of_the_names_counts_as_observed(monkeypatch):
    for i in range(len(fused._PROBES)):
        monkeypatch.setattr(fused, "_PROBES", fused._PROBES[:i] + (None,) + fused._PROBES[i + 1:])
        assert fused._observed()
        monkeypatch.undo()
    monkeypatch.delattr(forward_ad, "_current_level")
    assert fused._observed()


def test_cpu_lookups_and_training_lookups_do_not_probe(monkeypatch):
    from ghost_flow_b200.nn import Embedding

    def probe():
        raise AssertionError("probed")

    monkeypatch.setattr(fused, "_observed", probe)
    e = Embedding(5, 8)
    e(torch.tensor([1, 2]))
    with torch.no_grad():
        e(torch.tensor([1, 2]))
