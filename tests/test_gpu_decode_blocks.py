"""Decode attention at the edges of its blocks (16 keys to a warp's block, 64 to a CTA's round, a ring of three) against fp64."""
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


@pytest.mark.parametrize("H,Hk", [(1, 1), (6, 2), (8, 1), (5, 5)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("splits", [1, 2, 7, None])
@pytest.mark.parametrize("offset", [0, 1])
def test_every_length_against_fp64(H, Hk, D, splits, offset):
    from ghost_flow_b200.ops import raw

    lens = [0, 1, 15, 16, 17, 63, 64, 65, 127, 192, 193, 300, 511]
    B, n = len(lens), 512
    g = torch.Generator(device="cuda").manual_seed(H * D)
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    # queries and caches that start off a 16-byte boundary (for one of the head sizes that always was allowed)
    q = mk(B * H * D + offset)[offset:].view(B, H * D)
    k, v = (mk(B * n * Hk * D + offset)[offset:].view(B, n, Hk * D) for _ in range(2))
    k[3, 5:] = 0
    got = raw.attn_decode(q, k, v, torch.tensor(lens, dtype=torch.int32, device="cuda"), B, H, Hk, D, splits=splits)
    want = _want(q, k, v, lens, H, Hk, D)
    # P is rounded to bf16 (2^-9 of each probability) and the result once more
    assert (got.double() - want).norm() / want.norm() < 5e-3
    assert torch.allclose(got.double(), want, rtol=2 ** -6, atol=2 ** -7)
    same = raw.attn_decode(q[:1], k[:1], v[:1], 77, 1, H, Hk, D, splits=splits)
    assert torch.allclose(same.double(), _want(q, k, v, [77], H, Hk, D), rtol=2 ** -6, atol=2 ** -7)
