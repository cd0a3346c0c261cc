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
    # the result is rounded to bf16 (2^-9 at most, 2^-9 / sqrt(3) x 1.5 over many); what rounds before it is 2^-17 or less
    assert (got.double() - want).norm() / want.norm() < 2e-3
    assert torch.allclose(got.double(), want, rtol=2 ** -6, atol=2 ** -7)
    same = raw.attn_decode(q[:1], k[:1], v[:1], 77, 1, H, Hk, D, splits=splits)
    assert torch.allclose(same.double(), _want(q, k, v, [77], H, Hk, D), rtol=2 ** -6, atol=2 ** -7)


@pytest.mark.parametrize("n", [2, 16, 130])
@pytest.mark.parametrize("splits", [1, 3])
@pytest.mark.parametrize("D", [64, 128])
def test_probabilities_are_not_rounded_to_bf16(n, splits, D):
    from ghost_flow_b200.ops import raw

    # keys in pairs that score nearly the same, with values of opposite sign: the result is a difference of probabilities, and
    # what their rounding left is not hidden behind the rounding of the result
    B, H = 4, 12
    g = torch.Generator(device="cuda").manual_seed(n)
    k = torch.randn(B, n // 2, 1, H * D, generator=g, device="cuda").repeat(1, 1, 2, 1)
    k[:, :, 1] += 0.02 * torch.randn(B, n // 2, H * D, generator=g, device="cuda")
    v = torch.randn(B, n // 2, 1, H * D, generator=g, device="cuda").bfloat16()
    k, v = k.bfloat16().view(B, n, H * D), torch.cat((v, -v), 2).view(B, n, H * D)
    q = torch.randn(B, H * D, generator=g, device="cuda").bfloat16()
    want = _want(q, k, v, [n] * B, H, H, D)
    got = raw.attn_decode(q, k, v, n, B, H, H, D, splits=splits).double()
    # bf16 of the result (2^-9); before it probabilities in two bf16 numbers (2^-18 of each) times |v| < 4, and fp32 scores and
    # exponentials (2^-22). Rounded once to bf16 they are off by 2^-9 of each.
    assert torch.allclose(got, want, rtol=2 ** -8, atol=2 ** -16)
