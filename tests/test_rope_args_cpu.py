"""Rotary tables that do not hold the positions asked for are refused on the host: the kernels index them without a bound."""
import pytest
import torch

from ghost_flow_b200 import ops
from ghost_flow_b200.ops.fused import check_rope_tables


def test_tables_that_fit_are_accepted():
    cos, sin = ops.rope_tables(10, 32)
    for S, pos in [(10, 0), (1, 9), (4, 6)]:
        check_rope_tables(torch.device("cpu"), S, 32, cos, sin, pos)


@pytest.mark.parametrize("S,D,pos,device", [(11, 32, 0, "cpu"), (1, 32, 10, "cpu"), (5, 32, 6, "cpu"), (1, 32, -1, "cpu"),
                                            (1, 64, 0, "cpu"), (1, 16, 0, "cpu"), (1, 32, 0, "cuda:0")])
def test_tables_that_do_not_are_refused(S, D, pos, device):
    cos, sin = ops.rope_tables(10, 32)
    with pytest.raises(ValueError):
        check_rope_tables(torch.device(device), S, D, cos, sin, pos)


def test_sin_counts_as_much_as_cos():
    cos, sin = ops.rope_tables(10, 32)
    for bad in (sin[:5], sin[:, :8], sin[0]):
        with pytest.raises(ValueError):
            check_rope_tables(torch.device("cpu"), 6, 32, cos, bad, 0)


@pytest.mark.parametrize("heads", [5, 7])
def test_packed_projection_of_another_head_count_is_refused(heads):
    cos, sin = ops.rope_tables(10, 16)
    qkv = torch.randn(1, 3, heads, 16)
    with pytest.raises(ValueError):
        ops.rope_qkv(qkv, 2, 2, cos, sin)
    kc = torch.zeros(1, 10, 2, 16)
    with torch.no_grad(), pytest.raises(ValueError):
        ops.rope_qkv_to_cache(qkv, 2, 2, cos, sin, kc, kc.clone())
