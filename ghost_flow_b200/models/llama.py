"""LLaMA-family decoder as ``nn.Module`` (autograd path; the hand-scheduled ZeRO-3 engine in
``parallel/zero3.py`` runs the same math with explicit kernels).

Class and preset names follow ghostflow-nn/src/llama.rs:37-552 (``LLaMAConfig``, ``RMSNorm``, ``RotaryEmbedding``,
``SwiGLU``, ``LLaMAAttention``, ``LLaMADecoderLayer``, ``LLaMAModel``, ``LLaMAForCausalLM.forward/generate``).
Deviations from the reference, on purpose: real causal attention with K and V (its attention is a
placeholder that drops them, llama.rs:319-331), grouped-query attention, no biases, a KV cache in
``generate`` (its doc promises one, the code re-runs the whole prefix), N(0, 0.02) initialisation.
"""
from __future__ import annotations

import torch

from .. import ops
from ..ops import raw
from ..nn.layers import Embedding, Linear, RMSNorm, SwiGLU
from ..nn.module import Module, ModuleList, plain_modules
from .configs import LLaMAConfig


class LLaMAAttention(Module):
    def __init__(self, cfg: LLaMAConfig, device=None, dtype=None):
        super().__init__()
        self.cfg = cfg
        hd = cfg.head_dim
        self.wqkv = Linear(cfg.hidden_size, (cfg.num_attention_heads + 2 * cfg.num_key_value_heads) * hd, False,
                           device, dtype)
        self.wo = Linear(cfg.num_attention_heads * hd, cfg.hidden_size, False, device, dtype)

    def forward(self, x, cos, sin, residual=None, cache=None, start_pos: int = 0):
        c = self.cfg
        B, S, _ = x.shape
        H, Hk, D = c.num_attention_heads, c.num_key_value_heads, c.head_dim
        qkv = self.wqkv(x).view(B, S, H + 2 * Hk, D)
        if cache is not None:
            # decoding: append to the cache and attend over everything seen so far
            kc, vc = cache
            kernels = x.is_cuda and x.dtype == torch.bfloat16 and D in (64, 128) and not torch.is_grad_enabled()
            if kernels and start_pos == 0 and S > 1:
                # prompt: nothing older than itself to attend to
                q, k, v = ops.rope_qkv(qkv, H, Hk, cos, sin, c.rope_interleaved, start_pos)
                kc[:, :S] = k
                vc[:, :S] = v
                o = ops.flash_attention(q, k, v, causal=True)
            elif kernels and S == 1:
                q = ops.rope_qkv_to_cache(qkv, H, Hk, cos, sin, kc, vc, c.rope_interleaved, start_pos)
                # one new token per sequence: the decode kernel streams the cache once (GQA groups share the reads)
                o = raw.attn_decode(q.reshape(B, H * D), kc.view(B, kc.shape[1], Hk * D), vc.view(B, vc.shape[1], Hk * D),
                                    start_pos + 1, B, H, Hk, D).view(B, 1, H, D)
            else:
                q = ops.rope_qkv_to_cache(qkv, H, Hk, cos, sin, kc, vc, c.rope_interleaved, start_pos)
                kk, vv = kc[:, :start_pos + S], vc[:, :start_pos + S]
                G = H // Hk
                qf = q.transpose(1, 2).float()
                kf = kk.transpose(1, 2).float().repeat_interleave(G, 1)
                vf = vv.transpose(1, 2).float().repeat_interleave(G, 1)
                s = qf @ kf.transpose(-1, -2) / (D ** 0.5)
                T = start_pos + S
                mask = torch.ones(S, T, dtype=torch.bool, device=x.device).tril(T - S)
                s = s.masked_fill(~mask, float("-inf"))
                o = (torch.softmax(s, -1) @ vf).transpose(1, 2).to(x.dtype)
        else:
            q, k, v = ops.rope_qkv(qkv, H, Hk, cos, sin, c.rope_interleaved, start_pos)
            o = ops.flash_attention(q, k, v, causal=True)
        return self.wo(o.reshape(B, S, H * D), residual)


def _weight(module):
    """A module's weight: its parameter without the search of an attribute, or what else bears the name."""
    p = module._parameters.get("weight")
    return module.weight if p is None else p


class LLaMADecoderLayer(Module):
    def __init__(self, cfg: LLaMAConfig, device=None, dtype=None):
        super().__init__()
        self.attn_norm = RMSNorm(cfg.hidden_size, cfg.rms_norm_eps, device, dtype)
        self.attn = LLaMAAttention(cfg, device, dtype)
        self.ffn_norm = RMSNorm(cfg.hidden_size, cfg.rms_norm_eps, device, dtype)
        self.mlp = SwiGLU(cfg.hidden_size, cfg.intermediate_size, False, device, dtype)

    def _decodes_in_one_call(self, x, cos, sin, cache, start_pos):
        """The operands of :func:`ops.raw.llama_decode_layer`, or ``None`` where the layer runs module by module: more than one
        token, a gradient, other types or layouts, modules that were replaced or carry hooks, and calls that something
        follows (tracing, transforms, modes), which would miss what happens inside."""
        if x.dim() != 3 or x.shape[1] != 1 or x.dtype is not torch.bfloat16 or not x.is_cuda or torch.is_grad_enabled() \
                or type(x) is not torch.Tensor or not 0 < x.shape[0] <= 64 or not isinstance(start_pos, int) \
                or ops.observed():            # before anything asks a tensor for its memory: transformed ones have none
            return None
        m = self._modules                    # a plain callable that stands for a module is not in here
        an, at, fn, mlp = m.get("attn_norm"), m.get("attn"), m.get("ffn_norm"), m.get("mlp")
        if not (type(an) is RMSNorm and type(at) is LLaMAAttention and type(fn) is RMSNorm and type(mlp) is SwiGLU):
            return None
        lin = at._modules.get("wqkv"), at._modules.get("wo"), mlp._modules.get("gate_up"), mlp._modules.get("down")
        for n in lin:
            if type(n) is not Linear or n.bias is not None:
                return None
        if not plain_modules(an, at, fn, mlp, *lin):
            return None
        c, (kc, vc), (B, _, hidden), dev = at.cfg, cache, x.shape, x.device
        H, Hk, D = c.num_attention_heads, c.num_key_value_heads, c.head_dim
        w = [_weight(n) for n in (an, lin[0], lin[1], fn, lin[2], lin[3])]
        inner = w[5].shape[1] if w[5].dim() == 2 else 0
        shapes = (hidden,), ((H + 2 * Hk) * D, hidden), (hidden, H * D), (hidden,), (2 * inner, hidden), (hidden, inner)
        if D not in (64, 128) or H % Hk or H // Hk > 8 or hidden % 8 or inner % 8 or inner == 0:
            return None
        for p, s in zip(w, shapes):
            if p.shape != s or p.dtype is not torch.bfloat16 or p.device != dev or not p.is_contiguous() or p.data_ptr() & 15 \
                    or type(p) not in (torch.Tensor, torch.nn.Parameter):
                return None
        if dev.index != torch.cuda.current_device() or not (x.is_contiguous() and x.data_ptr() & 15 == 0) \
                or not ops.decode_cache_ok(kc, vc, cos, sin, (B, Hk, D), dev, start_pos):
            return None
        return (x, w[0], an.eps, w[1], w[2], w[3], fn.eps, w[4], w[5], cos, sin, kc, vc, H, Hk, D,
                c.rope_interleaved, start_pos)

    def forward(self, x, cos, sin, cache=None, start_pos: int = 0):
        if cache is not None:
            args = self._decodes_in_one_call(x, cos, sin, cache, start_pos)
            if args is not None:
                y = raw.llama_decode_layer(*args)
                torch.autograd.graph.increment_version(cache)     # a graph that saved a cache has to notice the write
                return y
        x = self.attn(self.attn_norm(x), cos, sin, residual=x, cache=cache, start_pos=start_pos)
        return self.mlp(self.ffn_norm(x), residual=x)


class LLaMAModel(Module):
    def __init__(self, cfg: LLaMAConfig, device=None, dtype=None):
        super().__init__()
        self.cfg = cfg
        self.embed_tokens = Embedding(cfg.vocab_size, cfg.hidden_size, device=device, dtype=dtype)
        self.layers = ModuleList([LLaMADecoderLayer(cfg, device, dtype) for _ in range(cfg.num_hidden_layers)])
        self.norm = RMSNorm(cfg.hidden_size, cfg.rms_norm_eps, device, dtype)
        self._rope = None

    def rope(self, length, device):
        if self._rope is None or self._rope[0].shape[0] < length or self._rope[0].device != torch.device(device):
            n = max(length, self.cfg.max_position_embeddings)
            self._rope = ops.rope_tables(n, self.cfg.head_dim, self.cfg.rope_theta, device)
        return self._rope

    def _before_norm(self, ids, caches, start_pos):
        S = ids.shape[1]
        cos, sin = self.rope(start_pos + S, ids.device)
        x = self.embed_tokens(ids)
        for i, layer in enumerate(self.layers):
            x = layer(x, cos, sin, None if caches is None else caches[i], start_pos)
        return x

    def forward(self, ids, caches=None, start_pos: int = 0):
        return self.norm(self._before_norm(ids, caches, start_pos))


class LLaMAForCausalLM(Module):
    def __init__(self, cfg: LLaMAConfig, device=None, dtype=None):
        super().__init__()
        self.cfg = cfg
        self.model = LLaMAModel(cfg, device, dtype)
        self.lm_head = Linear(cfg.hidden_size, cfg.vocab_size, False, device, dtype)
        self.reset_parameters()

    @torch.no_grad()
    def reset_parameters(self):
        std = self.cfg.initializer_range
        for name, p in self.named_parameters():
            if name.endswith("norm.weight"):
                p.fill_(1.0)
            else:
                p.normal_(0.0, std)
        if self.cfg.tie_word_embeddings:
            self.lm_head.weight = self.model.embed_tokens.weight

    def _norm_in_the_head(self, ids) -> bool:
        """Whether the last norm can run inside the head's product: one token of at most 16 sequences, no gradient, modules that do
        nothing but their own forward, dense bf16 weights on the current GPU, and nothing that follows the calls."""
        model, head = self._modules.get("model"), self._modules.get("lm_head")
        if type(ids) is not torch.Tensor or not ids.is_cuda or ids.dim() != 2 or ids.shape[1] != 1 or not 0 < ids.shape[0] <= 16 \
                or torch.is_grad_enabled() or ops.observed() or type(model) is not LLaMAModel or type(head) is not Linear \
                or head.bias is not None:
            return False
        norm, w = model._modules.get("norm"), head.weight
        if type(norm) is not RMSNorm or not plain_modules(model, norm, head) or ids.device.index != torch.cuda.current_device():
            return False
        for p, s in ((norm.weight, (self.cfg.hidden_size,)), (w, (w.shape[0], self.cfg.hidden_size))):
            if type(p) not in (torch.Tensor, torch.nn.Parameter) or p.shape != s or p.dtype is not torch.bfloat16 \
                    or p.device != ids.device or not p.is_contiguous() or p.data_ptr() & 15:
                return False
        return self.cfg.hidden_size % 8 == 0

    def forward(self, ids, labels=None, caches=None, start_pos: int = 0):
        if labels is None and caches is not None and self._norm_in_the_head(ids):
            x = self.model._before_norm(ids, caches, start_pos)
            if x.dtype is torch.bfloat16 and x.is_contiguous() and not x.data_ptr() & 15:
                norm, w = self.model.norm, self.lm_head.weight
                y = raw.rmsnorm_gemm(x.view(x.shape[0], -1), norm.weight, norm.eps, w)
                return y.unsqueeze(1)
            return self.lm_head(self.model.norm(x))
        h = self.model(ids, caches, start_pos)
        logits = self.lm_head(h)
        if labels is None:
            return logits
        return ops.cross_entropy(logits.view(-1, logits.shape[-1]), labels.reshape(-1)), logits

    def new_caches(self, batch: int, max_len: int, device=None, dtype=None):
        c = self.cfg
        p = next(self.parameters())
        shape = (batch, max_len, c.num_key_value_heads, c.head_dim)
        return [(torch.zeros(shape, device=device or p.device, dtype=dtype or p.dtype),
                 torch.zeros(shape, device=device or p.device, dtype=dtype or p.dtype))
                for _ in range(c.num_hidden_layers)]

    @torch.no_grad()
    def generate(self, ids, max_new_tokens: int, temperature: float = 0.0):
        """Greedy (temperature 0) or sampled continuation with a KV cache."""
        B, S = ids.shape
        caches = self.new_caches(B, S + max_new_tokens)
        logits = self.forward(ids, caches=caches, start_pos=0)[:, -1]
        out = [ids]
        pos = S
        for _ in range(max_new_tokens):
            if temperature and temperature > 0:
                nxt = torch.multinomial(torch.softmax(logits.float() / temperature, -1), 1)
            else:
                nxt = logits.argmax(-1, keepdim=True)
            out.append(nxt)
            logits = self.forward(nxt, caches=caches, start_pos=pos)[:, -1]
            pos += 1
        return torch.cat(out, dim=1)

    # names used by the ZeRO engine's state_dict
    def load_engine_state(self, sd: dict):
        """Loads the flat-unit names of ``Zero3LlamaEngine.state_dict()``."""
        own = self.state_dict()
        own["model.embed_tokens.weight"].copy_(sd["embed_tokens.weight"])
        own["model.norm.weight"].copy_(sd["norm.weight"])
        own["lm_head.weight"].copy_(sd["lm_head.weight"])
        for i in range(self.cfg.num_hidden_layers):
            pre = f"model.layers.{i}."
            own[pre + "attn_norm.weight"].copy_(sd[f"layers.{i}.attn_norm"])
            own[pre + "attn.wqkv.weight"].copy_(sd[f"layers.{i}.wqkv"])
            own[pre + "attn.wo.weight"].copy_(sd[f"layers.{i}.wo"])
            own[pre + "ffn_norm.weight"].copy_(sd[f"layers.{i}.ffn_norm"])
            own[pre + "mlp.gate_up.weight"].copy_(sd[f"layers.{i}.w_gate_up"])
            own[pre + "mlp.down.weight"].copy_(sd[f"layers.{i}.w_down"])
