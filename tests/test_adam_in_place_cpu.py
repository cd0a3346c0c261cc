"""Which parameter groups Adam may update in one launch that reads gradients and writes weights where they lie."""
import pytest
import torch

from ghost_flow_b200.ops import _lib
from ghost_flow_b200.ops.optim_kernels import adam_table
from ghost_flow_b200.optim.optimizers import Optimizer

BF = torch.bfloat16


def _group(params, grads, views=None):
    offs, n = [], 0
    for p in params:
        offs.append(n)
        n += (p.numel() + 3) // 4 * 4
    for p, g in zip(params, grads):
        p.grad = g
    return {"params": params, "offs": offs, "master": torch.zeros(n), "state": [torch.zeros(n) for _ in range(2)],
            "repeats": False, "is_view": views or [False] * len(params)}


def _in_place(f):
    """Whether the one launch takes the group: layouts first, then the library's check of the memory (no GPU needed)."""
    found = Optimizer._tensors_in_place(f)
    if found is None:
        return False
    return not _lib.cuda_lib().gf_adam_table_overlaps(f["master"].data_ptr(), *(s.data_ptr() for s in f["state"]), *adam_table(*found))


def _p(t):
    return torch.nn.Parameter(t)


def _ones(n):
    return torch.ones(n, dtype=BF)


def test_separate_tensors_and_shared_gradients_go_in_place():
    buf, g = _ones(64), _ones(16)
    ps = [_p(buf[:16]), _p(buf[16:32]), _p(buf[48:])]        # neighbours in one buffer
    f = _group(ps, [g, g, None])
    got, beside = Optimizer._tensors_in_place(f)
    assert [(id(a), id(b), o) for a, b, o in got] == [(id(g), id(ps[0]), 0), (id(g), id(ps[1]), 16)]
    assert len(beside) == 1 and beside[0] is ps[2] and _in_place(f)


@pytest.mark.parametrize("lo", [0, 1, 8, 15])
@pytest.mark.parametrize("second_has_grad", [True, False])
@pytest.mark.parametrize("order", [1, -1])
def test_overlapping_weights_take_the_flat_path(lo, second_has_grad, order):
    buf = _ones(64)
    ps = [_p(buf[:16]), _p(buf[lo:lo + 16])][::order]
    assert not _in_place(_group(ps, [_ones(16), _ones(16) if second_has_grad else None]))


@pytest.mark.parametrize("inner", [(4, 6), (0, 64)])
def test_a_weight_inside_another_takes_the_flat_path(inner):
    buf = _ones(64)
    ps = [_p(buf), _p(_ones(8)), _p(buf[inner[0]:inner[1]])]
    assert not _in_place(_group(ps, [torch.ones_like(p) for p in ps]))


def test_a_gradient_over_a_weight_or_the_flat_buffers_takes_the_flat_path():
    buf = _ones(64)
    ps = [_p(buf[:16]), _p(_ones(16))]
    for lo, ok in [(0, False), (15, False), (16, True)]:
        assert _in_place(_group(ps, [_ones(16), buf[lo:lo + 16]])) == ok
    f = _group([_p(torch.ones(16)), _p(torch.ones(16))], [torch.ones(16), torch.ones(16)], [True, True])
    assert _in_place(f)
    for b in (f["master"], *f["state"]):
        f["params"][0].grad = b[16:]
        assert not _in_place(f)


def test_other_layouts_take_the_flat_path():
    p = _p(torch.ones(4))
    assert not _in_place(_group([p], [torch._neg_view(torch.ones(4))], [True]))          # lazily negated
    p = _p(torch.ones(4, 6, dtype=BF))
    assert not _in_place(_group([p], [torch.ones(6, 4, dtype=BF).t()]))
    p = _p(torch.ones(6, 4, dtype=BF).t())
    assert not _in_place(_group([p], [torch.ones(4, 6, dtype=BF)]))
    p = _p(torch.ones(4, dtype=torch.float16))
    assert not _in_place(_group([p], [torch.ones(4, dtype=torch.float16)]))
