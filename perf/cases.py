"""The work whose speed this framework is judged by: the calls that a program training or serving a language model
makes, layer by layer, through the public entry points, over the sizes of the configurations in
``models/configs.py`` and of the benchmarks.

A case is a dict of plain values; ``kind`` names the call, the rest are its sizes. ``listed()`` gives the twelve
that stand for the ranges, ``draw(rng)`` another one of the same ranges.
"""
from __future__ import annotations

import math

import torch

BF16 = torch.bfloat16


# ------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # attention of one LLaMA-7B layer in training: the headline sequence of 4096 tokens, packed q, k, v, both directions
        dict(name="attention_train_4096", kind="attention_train", batch=1, seq=4096, heads=32, kv_heads=32, dim=128,
             causal=True),
        # attention of one GPT-2 layer in training, head dimension 64, batch of eight
        dict(name="attention_train_gpt2", kind="attention_train", batch=8, seq=1024, heads=12, kv_heads=12, dim=64,
             causal=True),
        # a prompt of odd length through grouped-query attention (8 query heads to a KV head), forward only
        dict(name="attention_prefill_odd", kind="attention_prefill", batch=2, seq=2987, heads=64, kv_heads=8, dim=128,
             causal=True),
        # one token of every sequence in a batch of mixed lengths over the KV cache
        dict(name="attention_decode", kind="attention_decode", batch=32, cache=4096, heads=32, kv_heads=8, dim=128),
        # one LLaMA-7B layer generating one token for eight sequences (weights are what is read)
        dict(name="llama_layer_decode", kind="llama_layer_decode", batch=8, pos=1500, hidden=4096, inner=11008, heads=32,
             kv_heads=32),
        # one LLaMA-7B layer, forward and backward, half the context
        dict(name="llama_layer_train", kind="llama_layer_train", batch=1, seq=2048, hidden=4096, inner=11008, heads=32,
             kv_heads=32),
        # one GPT-2 block (LayerNorm, biases, GELU), forward and backward
        dict(name="gpt2_block_train", kind="gpt_block_train", batch=8, seq=1024, hidden=768, inner=3072, heads=12),
        # RMSNorm with the residual add in front of it, forward and backward
        dict(name="rms_norm_train", kind="rms_norm_train", rows=8192, dim=4096, residual=True),
        # the loss over the GPT-2 vocabulary (odd, rows padded as the output head leaves them), with its gradient
        dict(name="loss_gpt2", kind="loss_train", rows=8192, vocab=50257, ignore=False),
        # one step of the optimizer over four blocks of GPT-2 medium, bf16 weights with fp32 masters
        dict(name="adamw_step", kind="adamw_step", blocks=4, hidden=1024, dtype="bf16"),
        # an e4m3 linear layer of LLaMA-7B (gate or up projection), forward and backward
        dict(name="fp8_linear_train", kind="fp8_linear_train", rows=4096, din=4096, dout=11008, bias=False),
        # the smallest call: a small model generating one token for three sequences
        dict(name="small_model_decode", kind="model_decode", batch=3, pos=40, layers=2, hidden=256, inner=512, heads=4,
             kv_heads=2, vocab=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _kv(rng, heads):
    return rng.choice([h for h in (heads, heads // 4, heads // 8) if h > 0 and heads % h == 0 and heads // h <= 8])


def draw(rng):
    kind = rng.choice(["attention_train", "attention_prefill", "attention_decode", "llama_layer_decode",
                       "llama_layer_train", "gpt_block_train", "rms_norm_train", "loss_train", "adamw_step",
                       "fp8_linear_train", "model_decode"])
    if kind == "attention_train":
        dim, heads = rng.choice([(64, 12), (64, 16), (64, 25), (128, 16), (128, 32), (128, 40)])
        seq = 128 * _log(rng, 1, 32)
        batch = max(1, min(_log(rng, 1, 16), 4096 * 4096 * 32 * 128 // (seq * seq * heads * dim)))
        causal = batch * seq * seq * heads * dim * 2 > 4096 * 4096 * 32 * 128 or rng.random() < 0.75
        return dict(kind=kind, batch=batch, seq=seq, heads=heads, kv_heads=_kv(rng, heads), dim=dim, causal=causal)
    if kind == "attention_prefill":
        dim, heads = rng.choice([(64, 12), (64, 16), (128, 16), (128, 32), (128, 64)])
        seq = _log(rng, 17, 4000)
        batch = max(1, min(_log(rng, 1, 16), 4096 * 4096 * 32 * 128 // (seq * seq * heads * dim)))
        return dict(kind=kind, batch=batch, seq=seq, heads=heads, kv_heads=_kv(rng, heads), dim=dim,
                    causal=rng.random() < 0.75)
    if kind == "attention_decode":
        dim, heads = rng.choice([(64, 12), (64, 16), (128, 32), (128, 40), (128, 64)])
        return dict(kind=kind, batch=_log(rng, 1, 64), cache=_log(rng, 64, 4096), heads=heads, kv_heads=_kv(rng, heads),
                    dim=dim)
    if kind in ("llama_layer_decode", "llama_layer_train"):
        hidden, inner, heads = rng.choice([(2048, 5504, 16), (4096, 11008, 32), (4096, 14336, 32), (5120, 13824, 40)])
        c = dict(kind=kind, hidden=hidden, inner=inner, heads=heads, kv_heads=_kv(rng, heads))
        if kind == "llama_layer_decode":
            return dict(c, batch=_log(rng, 1, 64), pos=_log(rng, 8, 2000))
        return dict(c, batch=1, seq=128 * _log(rng, 1, 10 if hidden > 4096 else 14))
    if kind == "gpt_block_train":
        hidden, heads = rng.choice([(768, 12), (1024, 16), (1280, 20), (1600, 25)])
        seq = 128 * _log(rng, 1, 8)
        return dict(kind=kind, batch=_log(rng, 1, 8192 // seq), seq=seq, hidden=hidden, inner=4 * hidden, heads=heads)
    if kind == "rms_norm_train":
        return dict(kind=kind, rows=_log(rng, 1, 16384), dim=8 * _log(rng, 16, 1024), residual=rng.random() < 0.5)
    if kind == "loss_train":
        return dict(kind=kind, rows=_log(rng, 16, 8192), vocab=rng.choice([1000, 30522, 32000, 50257]),
                    ignore=rng.random() < 0.5)
    if kind == "adamw_step":
        return dict(kind=kind, blocks=rng.randint(1, 5), hidden=64 * _log(rng, 2, 25), dtype=rng.choice(["bf16", "fp32"]))
    if kind == "fp8_linear_train":
        return dict(kind=kind, rows=16 * _log(rng, 8, 256), din=16 * _log(rng, 32, 256), dout=16 * _log(rng, 32, 688),
                    bias=rng.random() < 0.5)
    return dict(kind=kind, batch=_log(rng, 1, 8), pos=_log(rng, 1, 500), layers=rng.randint(1, 4),
                hidden=rng.choice([256, 512]), inner=rng.choice([512, 1376]), heads=4, kv_heads=rng.choice([2, 4]),
                vocab=rng.choice([512, 1000]))


# ------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, std=1.0, dtype=BF16):
    return (torch.randn(*shape, generator=g, device="cuda") * std).to(dtype)


def _norm_weight(g, n):
    return (1.0 + 0.1 * torch.randn(n, generator=g, device="cuda")).to(BF16)


def _llama_config(c):
    from ghost_flow_b200.models import LLaMAConfig

    return LLaMAConfig(vocab_size=c.get("vocab", 32000), hidden_size=c["hidden"], intermediate_size=c["inner"],
                       num_hidden_layers=c.get("layers", 1), num_attention_heads=c["heads"],
                       num_key_value_heads=c["kv_heads"], max_position_embeddings=4096)


def _llama_layer_weights(c, g):
    h, f = c["hidden"], c["inner"]
    d = h // c["heads"]
    return [_norm_weight(g, h), _randn(g, (c["heads"] + 2 * c["kv_heads"]) * d, h, std=0.02),
            _randn(g, h, c["heads"] * d, std=0.02), _norm_weight(g, h), _randn(g, 2 * f, h, std=0.02),
            _randn(g, h, f, std=0.02)]


def _llama_layer_params(m):
    return [m.attn_norm.weight, m.attn.wqkv.weight, m.attn.wo.weight, m.ffn_norm.weight, m.mlp.gate_up.weight,
            m.mlp.down.weight]


def _llama_layer(c, weights):
    from ghost_flow_b200.models.llama import LLaMADecoderLayer

    with torch.device("meta"):
        m = LLaMADecoderLayer(_llama_config(c), dtype=BF16)
    m = m.to_empty(device="cuda")
    with torch.no_grad():
        for p, w in zip(_llama_layer_params(m), weights):
            p.copy_(w)
    return m


def _gpt_weights(c, g):
    h, f = c["hidden"], c["inner"]
    return dict(ln1_w=_norm_weight(g, h), ln1_b=_randn(g, h, std=0.1), qkv_w=_randn(g, 3 * h, h, std=0.02),
                qkv_b=_randn(g, 3 * h, std=0.1), out_w=_randn(g, h, h, std=0.02), out_b=_randn(g, h, std=0.1),
                ln2_w=_norm_weight(g, h), ln2_b=_randn(g, h, std=0.1), fc1_w=_randn(g, f, h, std=0.02),
                fc1_b=_randn(g, f, std=0.1), fc2_w=_randn(g, h, f, std=0.02), fc2_b=_randn(g, h, std=0.1))


def _gpt_params(m):
    return dict(ln1_w=m.ln1.weight, ln1_b=m.ln1.bias, qkv_w=m.attn.qkv.weight, qkv_b=m.attn.qkv.bias,
                out_w=m.attn.out_proj.weight, out_b=m.attn.out_proj.bias, ln2_w=m.ln2.weight, ln2_b=m.ln2.bias,
                fc1_w=m.mlp.fc1.weight, fc1_b=m.mlp.fc1.bias, fc2_w=m.mlp.fc2.weight, fc2_b=m.mlp.fc2.bias)


def _block_shapes(h):
    return [(h,), (h,), (3 * h, h), (3 * h,), (h, h), (h,), (h,), (h,), (4 * h, h), (4 * h,), (h, 4 * h), (h,)]


def _inputs(c, seed):
    """The tensors of a case, from the seed alone (``exact`` makes the same ones)."""
    g, k = _gen(seed), c["kind"]
    if k in ("attention_train", "attention_prefill"):
        B, S, H, Hk, D = c["batch"], c["seq"], c["heads"], c["kv_heads"], c["dim"]
        s = dict(qkv=_randn(g, B, S, H + 2 * Hk, D))
        if k == "attention_train":
            s["do"] = _randn(g, B, S, H, D)
        return s
    if k == "attention_decode":
        B, n, H, Hk, D = c["batch"], c["cache"], c["heads"], c["kv_heads"], c["dim"]
        return dict(q=_randn(g, B, H * D), kc=_randn(g, B, n, Hk * D), vc=_randn(g, B, n, Hk * D),
                    lens=torch.randint(1, n + 1, (B,), generator=g, device="cuda", dtype=torch.int32))
    if k in ("llama_layer_train", "llama_layer_decode"):
        S = c["seq"] if k == "llama_layer_train" else 1
        s = dict(weights=_llama_layer_weights(c, g), x=_randn(g, c["batch"], S, c["hidden"]))
        if k == "llama_layer_train":
            s["dy"] = _randn(g, c["batch"], S, c["hidden"])
        else:
            shape = (c["batch"], c["pos"] + 64, c["kv_heads"], c["hidden"] // c["heads"])
            s["cache"] = (_randn(g, *shape), _randn(g, *shape))
        return s
    if k == "gpt_block_train":
        return dict(weights=_gpt_weights(c, g), x=_randn(g, c["batch"], c["seq"], c["hidden"]),
                    dy=_randn(g, c["batch"], c["seq"], c["hidden"]))
    if k == "rms_norm_train":
        s = dict(x=_randn(g, c["rows"], c["dim"]), w=_norm_weight(g, c["dim"]), dy=_randn(g, c["rows"], c["dim"]))
        if c["residual"]:
            s.update(res=_randn(g, c["rows"], c["dim"]), dh=_randn(g, c["rows"], c["dim"]))
        return s
    if k == "loss_train":
        T, V = c["rows"], c["vocab"]
        # the output head leaves rows that start on 16-byte boundaries whatever the vocabulary
        buf = torch.zeros(T, V if V % 8 == 0 else (V + 63) // 64 * 64, device="cuda", dtype=BF16)
        for lo in range(0, T, 1024):
            n = min(1024, T - lo)
            buf[lo:lo + n, :V] = _randn(g, n, V, std=2.0)
        tg = torch.randint(0, V, (T,), generator=g, device="cuda")
        if c["ignore"]:
            tg = tg.masked_fill(torch.rand(T, generator=g, device="cuda") < 0.2, -100)
            tg[0] = 1
        return dict(logits=buf[:, :V], targets=tg)
    if k == "adamw_step":
        dt = BF16 if c["dtype"] == "bf16" else torch.float32
        shapes = _block_shapes(c["hidden"]) * c["blocks"]
        return dict(params=[_randn(g, *s, std=0.05, dtype=dt) for s in shapes],
                    grads=[_randn(g, *s, std=1e-3, dtype=dt) for s in shapes])
    if k == "fp8_linear_train":
        s = dict(x=_randn(g, c["rows"], c["din"]), w=_randn(g, c["dout"], c["din"], std=0.02),
                 dy=_randn(g, c["rows"], c["dout"]))
        if c["bias"]:
            s["b"] = _randn(g, c["dout"], std=0.1)
        return s
    if k == "model_decode":
        shape = (c["batch"], c["pos"] + 16, c["kv_heads"], c["hidden"] // c["heads"])
        return dict(embed=_randn(g, c["vocab"], c["hidden"]), head=_randn(g, c["vocab"], c["hidden"], std=0.05),
                    norm=_norm_weight(g, c["hidden"]), layers=[_llama_layer_weights(c, g) for _ in range(c["layers"])],
                    ids=torch.randint(0, c["vocab"], (c["batch"], 1), generator=g, device="cuda"),
                    caches=[(_randn(g, *shape), _randn(g, *shape)) for _ in range(c["layers"])])
    raise ValueError(k)


def prepare(case, seed):
    from ghost_flow_b200 import ops
    from ghost_flow_b200.models import LLaMAForCausalLM
    from ghost_flow_b200.models.configs import GPTConfig
    from ghost_flow_b200.models.gpt import GPTBlock
    from ghost_flow_b200.optim import AdamW

    c, k = case, case["kind"]
    s = _inputs(c, seed)
    s["case"] = c
    if k == "attention_train":
        s["qkv"].requires_grad_(True)
    elif k in ("llama_layer_train", "llama_layer_decode"):
        s["layer"] = _llama_layer(c, s.pop("weights"))
        s["rope"] = ops.rope_tables(4096, c["hidden"] // c["heads"], 10000.0, "cuda")
        if k == "llama_layer_train":
            s["x"].requires_grad_(True)
    elif k == "gpt_block_train":
        cfg = GPTConfig(n_embd=c["hidden"], n_head=c["heads"], n_inner=c["inner"], dropout=0.0)
        with torch.device("meta"):
            m = GPTBlock(cfg)
        m = m.to(BF16).to_empty(device="cuda")
        w = s.pop("weights")
        with torch.no_grad():
            for n, p in _gpt_params(m).items():
                p.copy_(w[n])
        s["layer"] = m
        s["x"].requires_grad_(True)
    elif k == "rms_norm_train":
        for n in ("x", "w", "res"):
            if n in s:
                s[n].requires_grad_(True)
    elif k == "loss_train":
        s["logits"].requires_grad_(True)
    elif k == "adamw_step":
        s["params"] = [torch.nn.Parameter(p) for p in s["params"]]
        for p, gr in zip(s["params"], s.pop("grads")):
            p.grad = gr
        s["opt"] = AdamW(s["params"], lr=1e-3, weight_decay=0.01)
    elif k == "fp8_linear_train":
        from ghost_flow_b200.ops.fp8 import Fp8TrainLinear

        m = Fp8TrainLinear(c["din"], c["dout"], c["bias"], device="cuda", dtype=BF16)
        with torch.no_grad():
            m.weight.copy_(s.pop("w"))
            if c["bias"]:
                m.bias.copy_(s.pop("b"))
        s["layer"] = m
        s["x"].requires_grad_(True)
    elif k == "model_decode":
        m = LLaMAForCausalLM(_llama_config(c), device="cuda", dtype=BF16)
        with torch.no_grad():
            m.model.embed_tokens.weight.copy_(s.pop("embed"))
            m.lm_head.weight.copy_(s.pop("head"))
            m.model.norm.weight.copy_(s.pop("norm"))
            for layer, ws in zip(m.model.layers, s.pop("layers")):
                for p, w in zip(_llama_layer_params(layer), ws):
                    p.copy_(w)
        m.model.rope(c["pos"] + 1, s["ids"].device)
        s["model"] = m
    return s


# ------------------------------------------------------------------------------------------ one pass
def run(state):
    from ghost_flow_b200 import ops
    from ghost_flow_b200.ops import raw

    c, s = state["case"], state
    k = c["kind"]
    if k == "attention_train":
        s["qkv"].grad = None
        q, kk, v = ops.split_qkv(s["qkv"], c["heads"], c["kv_heads"])
        o = ops.flash_attention(q, kk, v, causal=c["causal"])
        o.backward(s["do"])
        return dict(o=o, dqkv=s["qkv"].grad)
    if k == "attention_prefill":
        q, kk, v = ops.split_qkv(s["qkv"], c["heads"], c["kv_heads"])
        return ops.flash_attention(q, kk, v, causal=c["causal"])
    if k == "attention_decode":
        return raw.attn_decode(s["q"], s["kc"], s["vc"], s["lens"], c["batch"], c["heads"], c["kv_heads"], c["dim"])
    if k == "llama_layer_decode":
        with torch.no_grad():
            y = s["layer"](s["x"], *s["rope"], cache=s["cache"], start_pos=c["pos"])
        return dict(y=y, k=s["cache"][0], v=s["cache"][1])
    if k in ("llama_layer_train", "gpt_block_train"):
        m = s["layer"]
        for p in m.parameters():
            p.grad = None
        s["x"].grad = None
        y = m(s["x"], *s["rope"]) if k == "llama_layer_train" else m(s["x"])
        y.backward(s["dy"])
        ps = _llama_layer_params(m) if k == "llama_layer_train" else list(_gpt_params(m).values())
        return dict(y=y, dx=s["x"].grad, dparams=[p.grad for p in ps])
    if k == "rms_norm_train":
        for n in ("x", "w", "res"):
            if n in s:
                s[n].grad = None
        if c["residual"]:
            y, h = ops.rms_norm(s["x"], s["w"], 1e-6, residual=s["res"])
            torch.autograd.backward([y, h], [s["dy"], s["dh"]])
            return dict(y=y, h=h, dx=s["x"].grad, dres=s["res"].grad, dw=s["w"].grad)
        y = ops.rms_norm(s["x"], s["w"], 1e-6)
        y.backward(s["dy"])
        return dict(y=y, dx=s["x"].grad, dw=s["w"].grad)
    if k == "loss_train":
        loss = ops.cross_entropy(s["logits"], s["targets"], ignore_index=-100 if c["ignore"] else None)
        (dl,) = torch.autograd.grad(loss, s["logits"])
        return dict(loss=loss, dlogits=dl)
    if k == "adamw_step":
        s["opt"].step()
        return list(s["params"])
    if k == "fp8_linear_train":
        m = s["layer"]
        for p in m.parameters():
            p.grad = None
        s["x"].grad = None
        y = m(s["x"])
        y.backward(s["dy"])
        return dict(y=y, dx=s["x"].grad, dparams=[p.grad for p in m.parameters()])
    if k == "model_decode":
        with torch.no_grad():
            return s["model"](s["ids"], caches=s["caches"], start_pos=c["pos"])
    raise ValueError(k)


# ------------------------------------------------------------------------------------------ the work of a pass
def _llama_layer_weight_count(c):
    h, f, d = c["hidden"], c["inner"], c["hidden"] // c["heads"]
    return (c["heads"] + 2 * c["kv_heads"]) * d * h + h * c["heads"] * d + 3 * f * h


def _pairs(S, causal):
    return S * (S + 1) / 2 if causal else float(S) * S


def work(case):
    c, k = case, case["kind"]
    if k in ("attention_train", "attention_prefill"):
        B, S, H, Hk, D = c["batch"], c["seq"], c["heads"], c["kv_heads"], c["dim"]
        qkv, o = 2.0 * B * S * (H + 2 * Hk) * D, 2.0 * B * S * H * D
        f = 4.0 * B * H * D * _pairs(S, c["causal"])
        return dict(bytes=2 * qkv + 2 * o, flops=3.5 * f) if k == "attention_train" else dict(bytes=qkv + o, flops=f)
    if k == "attention_decode":
        rows = c["batch"] * (c["cache"] + 1) / 2          # lengths are uniform over the cache
        return dict(bytes=4.0 * rows * c["kv_heads"] * c["dim"] + 4.0 * c["batch"] * c["heads"] * c["dim"],
                    flops=4.0 * rows * c["heads"] * c["dim"])
    if k in ("llama_layer_decode", "model_decode"):
        n, layers = _llama_layer_weight_count(c), c.get("layers", 1)
        d = c["hidden"] // c["heads"]
        kv = 4.0 * c["batch"] * (c["pos"] + 1) * c["kv_heads"] * d
        head = c["vocab"] * c["hidden"] if k == "model_decode" else 0
        return dict(bytes=layers * (2.0 * n + kv) + 2.0 * head + 4.0 * c["batch"] * c["hidden"],
                    flops=2.0 * c["batch"] * (layers * n + head) + layers * 4.0 * c["batch"] * (c["pos"] + 1) * c["hidden"])
    if k in ("llama_layer_train", "gpt_block_train"):
        h, T = c["hidden"], c["batch"] * c["seq"]
        n = _llama_layer_weight_count(c) if k == "llama_layer_train" else 4 * h * h + 2 * h * c["inner"]
        attn = 4.0 * c["batch"] * h * _pairs(c["seq"], True)
        return dict(bytes=4.0 * n + 8.0 * T * h, flops=6.0 * n * T + 3.5 * attn)
    if k == "rms_norm_train":
        n = float(c["rows"]) * c["dim"]
        # forward x (res) -> y (h); backward h, dy (dh) -> dx
        return dict(bytes=2.0 * n * (9 if c["residual"] else 5), flops=12.0 * n)
    if k == "loss_train":
        n = float(c["rows"]) * c["vocab"]
        return dict(bytes=4.0 * n, flops=6.0 * n)
    if k == "adamw_step":
        n = c["blocks"] * sum(math.prod(s) for s in _block_shapes(c["hidden"]))
        # fp32 master and two moments read and written, gradient read, bf16 weights written
        return dict(bytes=n * (24.0 + (4.0 if c["dtype"] == "bf16" else 4.0)), flops=14.0 * n)
    if k == "fp8_linear_train":
        T, K, N = c["rows"], c["din"], c["dout"]
        return dict(bytes=2.0 * (2 * T * K + 2 * T * N + 2 * N * K), flops=6.0 * T * K * N)
    raise ValueError(k)


def tolerance(case):
    k = case["kind"]
    # one kernel in front of a bf16 store: the store's own rounding (2^-9 at most, about 0.0017 over a whole result) on
    # both sides; attention also rounds its probabilities and their gradients to bf16
    if k in ("rms_norm_train", "loss_train"):
        return {"rel": 5e-3, "max": 0.05}
    if k in ("attention_train", "attention_prefill", "attention_decode"):
        return {"rel": 8e-3, "max": 0.1}
    if k == "adamw_step":
        return {"rel": 5e-3, "max": 0.05} if case["dtype"] == "bf16" else {"rel": 2e-6, "max": 1e-4}
    # layers: every intermediate tensor is stored in bf16, so roundings add up along the chain; e4m3 values may also fall
    # on the other side of a rounding boundary (a step of 1/8 of the value) where a scale differs in its last bit
    if k == "fp8_linear_train":
        return {"rel": 1e-2, "max": 0.2}
    return {"rel": 1.2e-2, "max": 0.25}


# ------------------------------------------------------------------------------------------ 64-bit results
def _f(t):
    return t.detach().double()


def _attn64(q, k, v, causal, lens=None):
    """q [B, S, H, D], k / v [B, T, Hk, D] in fp64, one (sequence, KV head) at a time."""
    B, S, H, D = q.shape
    T, Hk = k.shape[1], k.shape[2]
    G = H // Hk
    out = []
    for b in range(B):
        n = T if lens is None else int(lens[b])
        heads = []
        for h in range(Hk):
            s = q[b, :, h * G:(h + 1) * G].transpose(0, 1) @ k[b, :n, h].t() / math.sqrt(D)
            if causal:
                s = s.masked_fill(~torch.ones(S, n, dtype=torch.bool, device=s.device).tril(n - S), float("-inf"))
            heads.append((torch.softmax(s, -1) @ v[b, :n, h]).transpose(0, 1))
        out.append(torch.cat(heads, 1))
    return torch.stack(out)


def _rms64(x, w, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _rope64(x, pos):
    half = x.shape[-1] // 2
    inv = 10000.0 ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    ang = (pos + torch.arange(x.shape[1], device=x.device, dtype=torch.float64))[:, None] * inv
    co, si = ang.cos()[:, None], ang.sin()[:, None]
    a, b = x[..., :half], x[..., half:]
    return torch.cat((a * co - b * si, b * co + a * si), -1)


def _llama_layer64(c, w, x, cache=None, pos=0):
    B, S, _ = x.shape
    H, Hk = c["heads"], c["kv_heads"]
    D = c["hidden"] // H
    q, k, v = (_rms64(x, w[0]) @ w[1].t()).view(B, S, H + 2 * Hk, D).split([H, Hk, Hk], 2)
    q, k = _rope64(q, pos), _rope64(k, pos)
    kv = None
    if cache is not None:
        kv = [cache[0].clone(), cache[1].clone()]
        kv[0][:, pos:pos + S], kv[1][:, pos:pos + S] = k, v
        k, v = kv[0][:, :pos + S], kv[1][:, :pos + S]
    x = x + _attn64(q, k, v, True).reshape(B, S, H * D) @ w[2].t()
    g, u = (_rms64(x, w[3]) @ w[4].t()).chunk(2, -1)
    return x + (torch.nn.functional.silu(g) * u) @ w[5].t(), kv


def _ln64(x, w, b):
    return torch.nn.functional.layer_norm(x, (x.shape[-1],), w, b, 1e-5)


def _gpt_block64(c, w, x):
    B, S, h = x.shape
    H = c["heads"]
    q, k, v = (_ln64(x, w["ln1_w"], w["ln1_b"]) @ w["qkv_w"].t() + w["qkv_b"]).view(B, S, 3 * H, h // H).split(H, 2)
    x = x + _attn64(q, k, v, True).reshape(B, S, h) @ w["out_w"].t() + w["out_b"]
    m = _ln64(x, w["ln2_w"], w["ln2_b"]) @ w["fc1_w"].t() + w["fc1_b"]
    return x + torch.nn.functional.gelu(m, approximate="tanh") @ w["fc2_w"].t() + w["fc2_b"]


def exact(case, seed):
    c, k = case, case["kind"]
    s = _inputs(c, seed)
    if k in ("attention_train", "attention_prefill"):
        H, Hk = c["heads"], c["kv_heads"]
        if k == "attention_prefill":
            return _attn64(*_f(s["qkv"]).split([H, Hk, Hk], 2), c["causal"])
        qkv = _f(s["qkv"]).requires_grad_(True)
        o = _attn64(*qkv.split([H, Hk, Hk], 2), c["causal"])
        (g,) = torch.autograd.grad(o, qkv, _f(s["do"]))
        return dict(o=o, dqkv=g)
    if k == "attention_decode":
        B, H, Hk, D = c["batch"], c["heads"], c["kv_heads"], c["dim"]
        o = _attn64(_f(s["q"]).view(B, 1, H, D), _f(s["kc"]).view(B, -1, Hk, D), _f(s["vc"]).view(B, -1, Hk, D), False,
                    s["lens"])
        return o.reshape(B, H * D)
    if k == "llama_layer_decode":
        y, kv = _llama_layer64(c, [_f(w) for w in s["weights"]], _f(s["x"]), [_f(t) for t in s["cache"]], c["pos"])
        return dict(y=y, k=kv[0], v=kv[1])
    if k in ("llama_layer_train", "gpt_block_train"):
        llama = k == "llama_layer_train"
        w = [_f(t) for t in (s["weights"] if llama else s["weights"].values())]
        x = _f(s["x"])
        for t in [x, *w]:
            t.requires_grad_(True)
        y = _llama_layer64(c, w, x)[0] if llama else _gpt_block64(c, dict(zip(s["weights"], w)), x)
        g = torch.autograd.grad(y, [x, *w], _f(s["dy"]))
        return dict(y=y, dx=g[0], dparams=list(g[1:]))
    if k == "rms_norm_train":
        x, w = _f(s["x"]).requires_grad_(True), _f(s["w"]).requires_grad_(True)
        if c["residual"]:
            # the sum is stored in bf16 and the stored value is what gets normalised
            h = (s["x"].detach() + s["res"].detach()).double().requires_grad_(True)
            y = _rms64(h, w)
            dx, dw = torch.autograd.grad(y, [h, w], _f(s["dy"]))
            dx = dx + _f(s["dh"])
            return dict(y=y, h=_f(s["x"]) + _f(s["res"]), dx=dx, dres=dx, dw=dw)
        y = _rms64(x, w)
        dx, dw = torch.autograd.grad(y, [x, w], _f(s["dy"]))
        return dict(y=y, dx=dx, dw=dw)
    if k == "loss_train":
        lg = _f(s["logits"]).requires_grad_(True)
        loss = torch.nn.functional.cross_entropy(lg, s["targets"], ignore_index=-100)
        (g,) = torch.autograd.grad(loss, lg)
        return dict(loss=loss, dlogits=g)
    if k == "adamw_step":
        out = []
        for p, gr in zip(s["params"], s["grads"]):
            p, gr = _f(p), _f(gr)
            m, v = 0.1 * gr, 0.001 * gr * gr
            out.append(p * (1 - 1e-3 * 0.01) - 1e-3 * (m / 0.1) / ((v / 0.001).sqrt() + 1e-8))
        return out
    if k == "fp8_linear_train":
        x, w, dy = _f(s["x"]), _f(s["w"]), _f(s["dy"])
        y = x @ w.t()
        d = [dy.t() @ x]
        if c["bias"]:
            y = y + _f(s["b"])
            d.append(dy.sum(0))
        return dict(y=y, dx=dy @ w, dparams=d)
    if k == "model_decode":
        x = _f(s["embed"])[s["ids"]]
        for w, kv in zip(s["layers"], s["caches"]):
            x, _ = _llama_layer64(c, [_f(t) for t in w], x, [_f(t) for t in kv], c["pos"])
        return _rms64(x, _f(s["norm"])) @ _f(s["head"]).t()
    return None
