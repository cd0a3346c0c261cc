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


def test_parts_of_sequences_of_mixed_lengths():
    from ghost_flow_b200.ops.raw import _decode_parts

    for D in (64, 128):
        slots = 148 * (2 if D > 64 else 4)
        for B in (1, 2, 7, 62, 1000):
            for Hkv in (1, 8, 32):
                for n in (1, 64, 65, 300, 4000, 100000):
                    p, units = _decode_parts(B, Hkv, n, D, 148, True), (n + 63) // 64
                    # slices of 64 keys or more, as many pieces as the merge is made for; or shares of long sequences
                    assert (1 <= p <= min(16, units)) if p > 0 else (units >= 32 and B * Hkv * units >= 40 * slots and -p * Hkv <= slots)


# sizes at which numbers of slices were timed on 148 SMs with uniform lengths, with those that took at most 8 % longer than the best
@pytest.mark.parametrize("B,Hkv,n,D,good", [
    (62, 8, 300, 128, {1}), (62, 8, 130, 64, {1}), (31, 8, 300, 128, {1}), (4, 8, 4000, 128, {5, 6, 7, 8}), (4, 8, 4000, 64, {5, 6, 7, 8}),
    (16, 2, 4000, 128, {5, 6, 7, 8, 10}), (8, 8, 4000, 64, {6, 7, 8}), (2, 8, 8000, 128, {8, 10, 12, 16}), (62, 8, 800, 64, {1}),
    (8, 32, 800, 128, {1}), (16, 32, 300, 128, {1})])
def test_mixed_lengths_where_the_choice_matters(B, Hkv, n, D, good):
    from ghost_flow_b200.ops.raw import _decode_parts

    assert _decode_parts(B, Hkv, n, D, 148, True) in good
