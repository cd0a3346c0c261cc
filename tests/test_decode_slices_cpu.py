"""Slices of the KV cache in decode attention: within their limits for all sizes, and the good choice where the choices differ."""
import pytest

from ghost_flow_b200.ops.raw import _even_slices


def test_limits_hold_for_all_sizes():
    for D in (64, 128):
        for sms in (1, 132, 148):
            for ctas in [*range(1, 40), 147, 148, 149, 295, 296, 297, 591, 592, 593, 1200, 100000]:
                for blocks in (1, 2, 3, 7, 31, 32, 33, 200, 5000):
                    s = _even_slices(ctas, blocks, D, sms)
                    assert 1 <= s <= min(32, blocks)


# sizes at which numbers of slices were timed on 148 SMs, with those that took at most 4 % longer than the best
@pytest.mark.parametrize("ctas,n,D,good", [
    (160, 4000, 128, {3, 5, 7}), (248, 4000, 128, {1}), (320, 4000, 128, {3, 4, 5, 6, 8}), (496, 1000, 128, {1}), (96, 300, 128, {1}),
    (144, 300, 64, {1}), (240, 4000, 64, {1, 4}), (636, 4000, 64, {2, 3, 4, 5, 6, 8}), (312, 1500, 64, {1}), (80, 4000, 128, {3})])
def test_choice_where_it_matters(ctas, n, D, good):
    assert _even_slices(ctas, (n + 127) // 128, D, 148) in good
