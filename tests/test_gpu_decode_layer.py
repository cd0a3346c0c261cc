"""A LLaMA decoder layer for one token in one call (``gf_llama_decode_layer``) against fp64 and against the modules one by one."""
import ctypes
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture
def calls(monkeypatch):
    """The calls of the one-call layer."""
    from ghost_flow_b200.ops import raw

    seen, real = [], raw.llama_decode_layer
    monkeypatch.setattr(raw, "llama_decode_layer", lambda *a: seen.append(a) or real(*a))
    return seen


def _layer(hidden, inner, heads, kv, seed, **kw):
    from ghost_flow_b200.models import LLaMAConfig
    from ghost_flow_b200.models.llama import LLaMADecoderLayer

    cfg = LLaMAConfig(vocab_size=64, hidden_size=hidden, intermediate_size=inner, num_hidden_layers=1, num_attention_heads=heads,
                      num_key_value_heads=kv, max_position_embeddings=4096, **kw)
    m = LLaMADecoderLayer(cfg, device="cuda", dtype=torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(seed)
    with torch.no_grad():
        for n, p in m.named_parameters():
            p.copy_(1 + 0.1 * torch.randn(p.shape, generator=g, device="cuda") if p.dim() == 1
                    else torch.randn(p.shape, generator=g, device="cuda") / math.sqrt(p.shape[1]))
    return m, cfg, g


def _want(m, cfg, x, kc, vc, cos, sin, pos):
    from ghost_flow_b200.ops.fused import rope_ref

    d = lambda t: t.detach().double()  # noqa: E731
    H, Hk, D, B = cfg.num_attention_heads, cfg.num_key_value_heads, cfg.head_dim, x.shape[0]
    norm = lambda t, n: t * torch.rsqrt(t.square().mean(-1, keepdim=True) + n.eps) * d(n.weight)  # noqa: E731
    q, k, v = (norm(d(x), m.attn_norm) @ d(m.attn.wqkv.weight).t()).view(B, 1, H + 2 * Hk, D).split([H, Hk, Hk], 2)
    q, k = (rope_ref(t.float(), cos, sin, cfg.rope_interleaved, pos).double() for t in (q, k))
    kk, vv = torch.cat((d(kc[:, :pos]), k), 1), torch.cat((d(vc[:, :pos]), v), 1)
    s = torch.einsum("bhd,bnhd->bhn", q[:, 0], kk.repeat_interleave(H // Hk, 2)) / math.sqrt(D)
    o = torch.einsum("bhn,bnhd->bhd", torch.softmax(s, -1), vv.repeat_interleave(H // Hk, 2)).reshape(B, 1, H * D)
    h = d(x) + o @ d(m.attn.wo.weight).t()
    g, u = (norm(h, m.ffn_norm) @ d(m.mlp.gate_up.weight).t()).chunk(2, -1)
    return h + (torch.nn.functional.silu(g) * u) @ d(m.mlp.down.weight).t(), k, v


# token tiles of 16 / 32 / 64; positions at the edges of the attention's 64-key units and where a head is cut into parts
@pytest.mark.parametrize("B,pos", [(1, 0), (3, 63), (16, 64), (17, 127), (32, 300), (33, 1), (64, 700), (2, 4000)])
@pytest.mark.parametrize("hidden,inner,heads,kv,kw", [
    (256, 512, 4, 2, {}), (512, 1376, 4, 1, {"rope_interleaved": True}), (1024, 1000, 8, 8, {}), (2048, 5504, 16, 2, {})])
def test_layer_matches_fp64_and_the_modules(B, pos, hidden, inner, heads, kv, kw, calls):
    from ghost_flow_b200 import ops
    from ghost_flow_b200.ops import _lib

    m, cfg, g = _layer(hidden, inner, heads, kv, B + pos, **kw)
    D = cfg.head_dim
    if D not in (64, 128):
        pytest.skip("head size without a kernel")
    cos, sin = ops.rope_tables(4096, D, 10000.0, "cuda")
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, kc, vc = mk(B, 1, hidden), mk(B, pos + 3, kv, D), mk(B, pos + 3, kv, D)
    kc2, vc2 = kc.clone(), vc.clone()
    want, k, v = _want(m, cfg, x, kc, vc, cos, sin, pos)
    keep = kc.clone()
    with torch.no_grad():
        version = kc._version
        y = m(x, cos, sin, cache=(kc, vc), start_pos=pos)
        assert kc._version > version and len(calls) == 1
        hook = m.mlp.register_forward_hook(lambda *a: None)          # module by module
        y2 = m(x, cos, sin, cache=(kc2, vc2), start_pos=pos)
        hook.remove()
        assert len(calls) == 1
    _lib.check_status()
    # a chain of bf16 tensors (norm, q k v, attention, sum, norm, gate and up, their product), each rounded by 2^-9
    err, err2 = ((t.double() - want).norm() / want.norm() for t in (y, y2))
    assert err < 8e-3 and err < 1.1 * err2 + 1e-4
    for c, new in ((kc, k), (vc, v)):
        assert (c[:, pos].double() - new[:, 0]).norm() / new.norm() < 5e-3
    kc[:, pos] = keep[:, pos]
    assert torch.equal(kc, keep)


def test_layer_in_a_cuda_graph_and_where_it_is_not_taken(calls):
    from ghost_flow_b200 import ops

    m, cfg, g = _layer(512, 1024, 4, 2, 0)
    cos, sin = ops.rope_tables(512, 128, 10000.0, "cuda")
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, kc, vc = mk(5, 1, 512), mk(5, 400, 2, 128), mk(5, 400, 2, 128)
    with torch.no_grad():
        want = m(x, cos, sin, cache=(kc, vc), start_pos=333)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = m(x, cos, sin, cache=(kc, vc), start_pos=333)
        for _ in range(3):
            y.zero_()
            graph.replay()
            assert torch.equal(y, want)
        assert len(calls) == 2
        # caches that share rows are refused as before, and so are positions outside of the tables
        with pytest.raises(RuntimeError):
            m(x, cos, sin, cache=(kc[:1].expand(5, -1, -1, -1), vc), start_pos=3)
        with pytest.raises(ValueError):
            m(x, cos, sin, cache=(mk(5, 600, 2, 128), mk(5, 600, 2, 128)), start_pos=512)
        # more tokens or sequences, a replaced module, weights that are no dense bf16 tensors
        m(mk(5, 2, 512), cos, sin, cache=(kc, vc), start_pos=3)
        m(mk(65, 1, 512), cos, sin, cache=(mk(65, 9, 2, 128), mk(65, 9, 2, 128)), start_pos=3)
        w = m.mlp.down.weight
        m.mlp.down.weight = torch.nn.Parameter(w.t().contiguous().t())
        m(x, cos, sin, cache=(kc, vc), start_pos=3)
        m.mlp.down = torch.nn.Linear(1024, 512, bias=False, device="cuda", dtype=torch.bfloat16)
        m.mlp.down.forward = lambda t, residual: torch.nn.functional.linear(t, w) + residual
        m(x, cos, sin, cache=(kc, vc), start_pos=3)
        assert len(calls) == 2
    m, cfg, g = _layer(512, 1024, 4, 2, 0)
    assert m(x, cos, sin, cache=(kc.clone(), vc.clone()), start_pos=3).requires_grad and len(calls) == 2


@pytest.mark.parametrize("vocab,B", [(64, 1), (1003, 3), (512, 16), (512, 17)])
def test_norm_inside_the_head(vocab, B, monkeypatch):
    """Logits of a decoding step with the last norm in front of the head's product, and module by module."""
    from ghost_flow_b200.models import LLaMAConfig, LLaMAForCausalLM
    from ghost_flow_b200.ops import raw

    cfg = LLaMAConfig(vocab_size=vocab, hidden_size=256, intermediate_size=512, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=2, max_position_embeddings=128)
    m = LLaMAForCausalLM(cfg, device="cuda", dtype=torch.bfloat16)
    g = torch.Generator(device="cuda").manual_seed(vocab)
    seen, real = [], raw.rmsnorm_gemm
    monkeypatch.setattr(raw, "rmsnorm_gemm", lambda *a: seen.append(a) or real(*a))
    ids = torch.randint(0, vocab, (B, 1), generator=g, device="cuda")
    with torch.no_grad():
        m.model.norm.weight.copy_(1 + 0.1 * torch.randn(256, generator=g, device="cuda"))
        mk = lambda: [tuple(torch.randn(B, 20, 2, 64, generator=torch.Generator(device="cuda").manual_seed(i), device="cuda")  # noqa: E731
                            .bfloat16() for _ in range(2)) for i in range(2)]
        y = m(ids, caches=mk(), start_pos=9)
        assert len(seen) == (1 if B <= 16 else 0) and y.shape == (B, 1, vocab)
        hidden = []
        hook = m.model.norm.register_forward_hook(lambda mod, a, out: hidden.append(a[0]))
        y2 = m(ids, caches=mk(), start_pos=9)
        hook.remove()
        assert len(seen) == (1 if B <= 16 else 0)
        x = hidden[0].double()
        want = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + m.model.norm.eps) * m.model.norm.weight.double()
        want = want @ m.lm_head.weight.double().t()
    # the operand is rounded once on either path, and the result
    e, e2 = ((t.double() - want).norm() / want.norm() for t in (y, y2))
    assert e < 4e-3 and e < 1.2 * e2 + 1e-4
    assert torch.equal(m.generate(ids, 3)[:, :2], m.generate(ids, 1))


def test_weights_and_modules_that_plain_attributes_replace(calls):
    """A weight put on a module as a tensor is a weight; a callable in the place of a module is called."""
    import copy

    from ghost_flow_b200 import ops
    from ghost_flow_b200.models import LLaMAForCausalLM

    m, cfg, g = _layer(256, 512, 4, 2, 3)
    cos, sin = ops.rope_tables(64, 64, 10000.0, "cuda")
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, caches = mk(2, 1, 256), (mk(2, 40, 2, 64), mk(2, 40, 2, 64))
    step = lambda l: l(x, cos, sin, cache=tuple(c.clone() for c in caches), start_pos=7)  # noqa: E731
    with torch.no_grad():
        want = step(m)
        for name in ("attn_norm", "attn.wqkv", "attn.wo", "ffn_norm", "mlp.gate_up", "mlp.down"):
            r = copy.deepcopy(m)
            n = r.get_submodule(name)
            w = n.weight.detach()
            del n.weight
            n.weight = w
            assert torch.equal(step(r), want), name
        taken = len(calls)
        for owner, name in (("", "attn_norm"), ("attn", "wqkv"), ("attn", "wo"), ("", "mlp"), ("mlp", "down")):
            r = copy.deepcopy(m)
            o = r.get_submodule(owner)
            real = getattr(o, name)
            delattr(o, name)
            setattr(o, name, lambda *a, real=real, **k: real(*a, **k))
            # roundings of a chain of bf16 tensors, as above
            assert ((step(r).float() - want.float()).norm() / want.float().norm()) < 8e-3, name
        assert len(calls) == taken

        lm = LLaMAForCausalLM(cfg, device="cuda", dtype=torch.bfloat16)
        ids = torch.randint(0, 64, (2, 1), generator=g, device="cuda")
        logits = lambda l: l(ids, caches=[tuple(c.clone() for c in caches)], start_pos=7).float()  # noqa: E731
        want = logits(lm)
        for owner, name in (("", "lm_head"), ("model", "norm")):
            r = copy.deepcopy(lm)
            o = r.get_submodule(owner)
            real = getattr(o, name)
            delattr(o, name)
            setattr(o, name, lambda *a, real=real: real(*a))
            assert (logits(r) - want).norm() / want.norm() < 8e-3, name


def test_positions_that_are_no_int_are_refused(calls):
    import numpy as np

    from ghost_flow_b200 import ops

    m, _, g = _layer(256, 512, 4, 2, 3)
    cos, sin = ops.rope_tables(64, 64, 10000.0, "cuda")
    x, kc, vc = (torch.randn(*s, generator=g, device="cuda").bfloat16() for s in ((2, 1, 256), (2, 40, 2, 64), (2, 40, 2, 64)))
    with torch.no_grad():
        for pos in (np.int64(7), torch.tensor(7), 7.0):
            with pytest.raises((TypeError, ctypes.ArgumentError)):
                m(x, cos, sin, cache=(kc, vc), start_pos=pos)
    assert not calls


def test_wide_inner_layer(calls):
    """More activations between the last two products than a thread of their kernel usually has vectors for."""
    from ghost_flow_b200 import ops
    from ghost_flow_b200.ops import _lib

    m, cfg, g = _layer(64, 131072, 1, 1, 5)
    cos, sin = ops.rope_tables(64, 64, 10000.0, "cuda")
    mk = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    x, kc, vc = mk(64, 1, 64), mk(64, 9, 1, 64), mk(64, 9, 1, 64)
    want, _, _ = _want(m, cfg, x, kc, vc, cos, sin, 7)
    with torch.no_grad():
        y = m(x, cos, sin, cache=(kc, vc), start_pos=7)
    _lib.check_status()
    assert len(calls) == 1 and (y.double() - want).norm() / want.norm() < 8e-3      # as above
