"""Many decoder layers and steps back to back: each layer's launches overlap with each other and its workspaces are used again by the next
ones, so what is read too early or overwritten too soon shows as a difference from the same calls one at a time."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _model(hidden, inner, heads, kv, layers, vocab, seed):
    from ghost_flow_b200.models import LLaMAConfig, LLaMAForCausalLM

    cfg = LLaMAConfig(vocab_size=vocab, hidden_size=hidden, intermediate_size=inner, num_hidden_layers=layers, num_attention_heads=heads,
                      num_key_value_heads=kv, max_position_embeddings=256)
    m = LLaMAForCausalLM(cfg, device="cuda", dtype=torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(seed)
    with torch.no_grad():
        for p in m.parameters():
            r = torch.randn(p.shape, generator=g, device="cuda")
            p.copy_(r / math.sqrt(p.shape[1]) if p.dim() == 2 else 1 + 0.1 * r)
    return m, g


def _decode(m, ids, steps, between):
    """Logits of every step and the caches at the end; the inputs change from step to step."""
    caches = m.new_caches(ids.shape[0], 128)
    out = []
    with torch.no_grad():
        for i in range(steps):
            out.append(m((ids + 7 * i) % m.cfg.vocab_size, caches=caches, start_pos=i))
            between()
    torch.cuda.synchronize()
    return torch.stack(out), caches


# the norm in front of a product or as a kernel, one or several pieces of a head's keys, the kernels with and without a merge
@pytest.mark.parametrize("B,hidden,inner,heads,kv,layers,steps", [
    (1, 256, 688, 4, 2, 32, 50), (3, 1024, 2816, 8, 8, 32, 70), (16, 512, 1376, 8, 1, 24, 50), (17, 256, 512, 4, 4, 24, 50), (64, 512, 1024, 4, 2, 8, 70)])
def test_steps_back_to_back_equal_steps_one_at_a_time(B, hidden, inner, heads, kv, layers, steps, kernel_status):
    m, g = _model(hidden, inner, heads, kv, layers, 512, B)
    ids = torch.randint(0, 512, (B, 1), generator=g, device="cuda")
    want, kv_want = _decode(m, ids, steps, torch.cuda.synchronize)
    # one launch after the other has ended: every layer waits, too
    hooks = [layer.register_forward_hook(lambda *a: torch.cuda.synchronize()) for layer in m.model.layers]
    alone, kv_alone = _decode(m, ids, steps, torch.cuda.synchronize)
    for h in hooks:
        h.remove()
    assert torch.equal(want, alone)
    for _ in range(3):
        got, kv_got = _decode(m, ids, steps, lambda: None)
        assert torch.equal(got, want)
        for a, b in zip(kv_got, kv_want):
            assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])


def test_two_streams_at_once(kernel_status):
    """Layers of two models on two streams: no workspace, flag or slot is shared."""
    (m, g), (n, _) = _model(512, 1376, 8, 2, 12, 512, 1), _model(256, 688, 4, 4, 16, 512, 2)
    ids = torch.randint(0, 512, (2, 1), generator=g, device="cuda")
    want = [_decode(t, ids, 40, torch.cuda.synchronize)[0] for t in (m, n)]
    streams = [torch.cuda.Stream() for _ in range(2)]
    caches = [t.new_caches(2, 128) for t in (m, n)]
    torch.cuda.synchronize()
    out = [[], []]
    with torch.no_grad():
        for i in range(40):
            for k, t in enumerate((m, n)):
                with torch.cuda.stream(streams[k]):
                    out[k].append(t((ids + 7 * i) % 512, caches=caches[k], start_pos=i))
    torch.cuda.synchronize()
    for k in range(2):
        assert torch.equal(torch.stack(out[k]), want[k])
