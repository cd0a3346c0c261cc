"""Attention backward (128-row steps) against the gradient in fp64: one and several query tiles, tile stages that wrap,
grouped heads, both head sizes, with and without a mask, heads of several sequences in one block order."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _exact(q, k, v, do, causal):
    q, k, v = (t.double().requires_grad_() for t in (q, k, v))
    S, G = q.shape[1], q.shape[2] // k.shape[2]
    kk, vv = k.repeat_interleave(G, 2), v.repeat_interleave(G, 2)
    s = torch.einsum("bqhd,bkhd->bhqk", q, kk) / math.sqrt(q.shape[-1])
    if causal:
        s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=s.device).tril(), float("-inf"))
    o = torch.einsum("bhqk,bkhd->bqhd", torch.softmax(s, -1), vv)
    return torch.autograd.grad(o, (q, k, v), do.double())


@pytest.mark.parametrize("B,S,H,Hk", [(1, 128, 1, 1), (3, 256, 3, 1), (2, 384, 4, 2), (1, 1152, 5, 5), (5, 640, 8, 1)])
@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_gradients_match_fp64(B, S, H, Hk, D, causal, kernel_status):
    from ghost_flow_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(B * S + H)
    q, k, v = (torch.randn(B, S, h, D, generator=g, device="cuda").bfloat16().requires_grad_() for h in (H, Hk, Hk))
    do = torch.randn(B, S, H, D, generator=g, device="cuda").bfloat16()
    o = ops.flash_attention(q, k, v, causal=causal)
    o.backward(do)
    for got, want in zip((q.grad, k.grad, v.grad), _exact(q.detach(), k.detach(), v.detach(), do, causal)):
        # P and dS are rounded to bf16 (2^-9) on their way into the products, the result once more. By row, so that a
        # missing or misplaced tile shows (it is off by the row's own size): a row that sees two or three keys takes
        # delta = O dO with O rounded to bf16, a random error of 2^-9 sqrt(D), into dQ as scale |k| = 1 times that, 0.02,
        # while the typical row of a long causal sequence is only about 0.3 long
        err = (got.double() - want).norm(dim=-1) / want.norm(dim=-1).clamp_min(want.norm() / math.sqrt(want[..., 0].numel()))
        assert err.max().item() < 0.1 and ((got.double() - want).norm() / want.norm()).item() < 5e-3


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("pad,shift", [(4, 0), (0, 4), (4, 4)])
def test_rows_on_8_byte_boundaries(D, pad, shift, kernel_status):
    """The caller's own pitch and offset for o and dq; same numbers as from packed rows."""
    from ghost_flow_b200.ops import raw

    B, S, H = 2, 256, 2
    g = torch.Generator(device="cuda").manual_seed(D + pad)
    q, k, v, do = (torch.randn(B * S, H * D, generator=g, device="cuda").bfloat16() for _ in range(4))
    o, lse = raw.attn_fwd(q, k, v, B, S, H, H, D)

    def strided(fill):
        t = torch.zeros(B * S * (H * D + pad) + shift, device="cuda", dtype=torch.bfloat16)[shift:].view(B * S, H * D + pad)
        return t, t[:, :H * D].copy_(fill)

    got = []
    for narrow in (False, True):
        whole, dq = strided(torch.zeros_like(q)) if narrow else (None, torch.empty_like(q))
        oo = strided(o)[1] if narrow else o
        raw.attn_bwd(q, k, v, oo, do, lse, dq, torch.empty_like(k), torch.empty_like(v), B, S, H, H, D)
        got.append(dq)
        if narrow and pad:
            assert whole[:, H * D:].count_nonzero().item() == 0
    # sums of two key tiles in either order, rounded once to bf16
    assert torch.allclose(got[0].float(), got[1].float(), rtol=2 ** -8, atol=1e-6)
