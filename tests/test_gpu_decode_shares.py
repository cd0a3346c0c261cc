"""Decode attention with the keys of all sequences cut into equal shares: parts that begin and end anywhere, against fp64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _want(q, k, v, lens, H, Hk, D):
    out = []
    for b, n in enumerate(lens):
        kk = k[b, :n].double().view(n, Hk, D).repeat_interleave(H // Hk, 1)
        vv = v[b, :n].double().view(n, Hk, D).repeat_interleave(H // Hk, 1)
        p = torch.softmax(torch.einsum("hd,nhd->hn", q[b].double().view(H, D), kk) / math.sqrt(D), -1)
        out.append(torch.einsum("hn,nhd->hd", p, vv).reshape(-1) if n else torch.zeros(H * D, device=q.device).double())
    return torch.stack(out)


# one part for everything, a few sequences to a part, sequences over more parts than the merge takes in one trip, more parts than
# units; more sequences than the scan of the lengths takes at a time
@pytest.mark.parametrize("parts", [1, 2, 7, 40, 1000])
@pytest.mark.parametrize("H,Hk,D", [(1, 1, 128), (6, 2, 64), (8, 1, 128), (5, 5, 64), (16, 2, 128)])
@pytest.mark.parametrize("lens", [[0, 1, 15, 64, 65, 300, 0, 511, 700], [700], [64, 0, 130] * 14])
def test_shares_of_all_sequences(parts, H, Hk, D, lens, monkeypatch):
    from ghost_flow_b200.ops import raw

    monkeypatch.setattr(raw, "_decode_parts", lambda *a: -parts)
    B, n = len(lens), 700
    g = torch.Generator(device="cuda").manual_seed(parts + H)
    q, k, v = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((B, H * D), (B, n, Hk * D), (B, n, Hk * D)))
    got = raw.attn_decode(q, k, v, torch.tensor(lens, dtype=torch.int32, device="cuda"), B, H, Hk, D)
    want = _want(q, k, v, lens, H, Hk, D)
    # the result is rounded to bf16, as with parts of each sequence; sums of pieces are fp32
    assert (got.double() - want).norm() / want.norm() < 2e-3
    assert torch.allclose(got.double(), want, rtol=2 ** -6, atol=2 ** -7)
    if len(set(lens)) == 1:
        assert torch.equal(got, raw.attn_decode(q, k, v, lens[0], B, H, Hk, D))


def test_which_calls_take_shares():
    from ghost_flow_b200.ops.raw import _decode_parts

    assert _decode_parts(32, 8, 4096, 128, 148, True) == -37 and _decode_parts(32, 12, 4096, 64, 148, True) == -49
    assert _decode_parts(32, 8, 4096, 128, 148, False) > 0 and _decode_parts(3, 8, 41, 128, 148, True) == 1
    for B, Hk, n, D in [(1, 1, 1, 64), (64, 32, 64, 64), (1, 64, 100000, 128), (600, 1, 5000, 128)]:
        p = _decode_parts(B, Hk, n, D, 148, True)
        assert 1 <= p <= 32 or 1 <= -p * Hk <= 148 * 4


def test_parts_below_one_are_refused():
    from ghost_flow_b200.ops import raw

    t = torch.zeros(1, 128, device="cuda", dtype=torch.bfloat16)
    c = torch.zeros(1, 4, 128, device="cuda", dtype=torch.bfloat16)
    for s in (0, -1):
        with pytest.raises(ValueError):
            raw.attn_decode(t, c, c, 4, 1, 1, 1, 128, splits=s)
