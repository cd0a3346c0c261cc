"""Block order of the forward attention kernel: heads of all sequences in groups that follow the size of K and V, with a
last group that is not full, and ragged query blocks, against fp64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


# (1, 5000, 10 / 5): 5 MB of K and V to two heads, so groups of eight and a last one of two; (3, 129..): groups across sequences
@pytest.mark.parametrize("B,S,H,Hk,D", [(1, 1, 1, 1, 64), (3, 129, 3, 3, 64), (5, 257, 6, 2, 128), (2, 255, 9, 3, 128),
                                        (1, 5000, 10, 5, 128), (1, 9000, 9, 9, 128)])
@pytest.mark.parametrize("causal", [True, False])
def test_every_query_row_of_every_head(B, S, H, Hk, D, causal):
    from ghost_flow_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v = (torch.randn(B, S, h, D, generator=g, device="cuda").bfloat16() for h in (H, Hk, Hk))
    o = ops.flash_attention(q, k, v, causal=causal)
    for b in range(B):
        for h in range(H):
            s = q[b, :, h].double() @ k[b, :, h // (H // Hk)].double().t() / math.sqrt(D)
            if causal:
                s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device="cuda").tril(), float("-inf"))
            want = torch.softmax(s, -1) @ v[b, :, h // (H // Hk)].double()
            # P and O are rounded to bf16 (2^-9 each); a wrong or missing block is off by its whole size
            rel = ((o[b, :, h].double() - want).norm(dim=-1) / want.norm(dim=-1).clamp_min(0.05)).max().item()
            assert rel < 2e-2, (b, h, rel)
