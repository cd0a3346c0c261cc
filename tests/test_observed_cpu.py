"""What counts as following the operations of a call (``ops.observed``)."""
import subprocess
import sys

import pytest
import torch
import torch.autograd.forward_ad as fwd_ad
from torch.overrides import TorchFunctionMode
from torch.utils._python_dispatch import TorchDispatchMode

from ghost_flow_b200 import ops


class _Function(TorchFunctionMode):
    def __torch_function__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


class _Dispatch(TorchDispatchMode):
    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        return func(*args, **(kwargs or {}))


def test_device_contexts_follow_nothing():
    assert not ops.observed()
    with torch.device("cpu"):
        assert not ops.observed()
        with torch.device("meta"):
            assert not ops.observed()
    code = "import torch; torch.set_default_device('cpu')\nfrom ghost_flow_b200 import ops\nassert not ops.observed()"
    subprocess.run([sys.executable, "-c", code], check=True)


@pytest.mark.parametrize("mode", [_Function, _Dispatch, fwd_ad.dual_level])
def test_modes_do(mode):
    with mode():
        assert ops.observed()
        with torch.device("cpu"):
            assert ops.observed()
    with torch.device("cpu"), mode():
        assert ops.observed()
    assert not ops.observed()


def test_tracing_and_transforms_do():
    seen = []
    f = lambda x: seen.append(ops.observed()) or x + 1  # noqa: E731
    x = torch.zeros(2)
    torch.jit.trace(f, (x,), check_trace=False)
    torch.func.vmap(f)(x)
    torch.func.jvp(f, (x,), (x,))
    assert seen == [True] * 3
