"""Explicit forward / backward primitives (no autograd graph) used by the hand-scheduled training
engines. Each primitive launches the sm_100a kernel for bf16 CUDA tensors and runs the same math
in PyTorch for CPU tensors, so the engines' partitioning and scheduling logic can be tested with
CPU ranks over gloo.
"""
from __future__ import annotations

import functools
import math

import torch
import torch.nn.functional as F

from . import _lib
from .fused import _scratch, check_rope_tables, rope_ref
from .gemm import _sm_count, gemm_raw


def _k(t: torch.Tensor) -> bool:
    return t.is_cuda and t.dtype == torch.bfloat16


def _rc(rc, what):
    _lib.check_rc(rc, what)


# ------------------------------------------------------------------ GEMM
def gemm(a, a_t: bool, b, b_t: bool, out=None, out_dtype=None, bias=None, residual=None, accumulate=False,
         alpha=1.0, **kw):
    """``op(a) @ op(b)`` with ``op(a) = a^T`` when ``a_t`` (a stored [K, M]) and ``op(b) = b^T`` when
    ``b_t`` (b stored [N, K], the usual weight layout)."""
    M = a.shape[1] if a_t else a.shape[0]
    K = a.shape[0] if a_t else a.shape[1]
    N = b.shape[0] if b_t else b.shape[1]
    if _k(a) and _k(b):
        return gemm_raw(a, a_t, b, not b_t, M, N, K, out=out,
                        out_dtype=out_dtype or torch.bfloat16, bias=bias, residual=residual,
                        accumulate=accumulate, alpha=alpha, **kw)
    af = (a.t() if a_t else a).float()
    bf = (b.t() if b_t else b).float()
    y = alpha * (af @ bf)
    if bias is not None:
        y = y + bias.float()
    if residual is not None:
        y = y + residual.float()
    if out is not None:
        if accumulate:
            y = y + out.float()
        out.copy_(y.to(out.dtype))
        return out
    return y.to(out_dtype or a.dtype)


# ------------------------------------------------------------------ RMSNorm
def rmsnorm_fwd(x, w, eps, residual=None):
    """Returns (y, rstd, h) where h = x + residual (or x itself when there is no residual)."""
    T, D = x.shape
    if _k(x):
        y = torch.empty_like(x)
        rstd = torch.empty(T, dtype=torch.float32, device=x.device)
        h = torch.empty_like(x) if residual is not None else x
        _rc(_lib.cuda_lib().gf_rmsnorm_fwd(x.data_ptr(), residual.data_ptr() if residual is not None else None,
                                           w.data_ptr(), y.data_ptr(),
                                           h.data_ptr() if residual is not None else None, rstd.data_ptr(), T, D,
                                           float(eps), _lib.stream_ptr()), "gf_rmsnorm_fwd")
        return y, rstd, h
    h = x if residual is None else (x.float() + residual.float()).to(x.dtype)
    hf = h.float()
    rstd = torch.rsqrt(hf.pow(2).mean(-1) + eps)
    y = (hf * rstd[:, None] * w.float()).to(x.dtype)
    return y, rstd, h


def rmsnorm_bwd(x, w, dy, rstd, dres=None, dw_out=None):
    """Returns (dx, dw). ``dres`` is added into dx; ``dw_out`` receives dw when given."""
    T, D = x.shape
    if _k(x):
        dx = torch.empty_like(x)
        dw = dw_out if dw_out is not None else torch.empty_like(w)
        lib = _lib.cuda_lib()
        g = lib.gf_norm_bwd_grid(T)
        scratch = _scratch(x.device, g * D)
        _rc(lib.gf_rmsnorm_bwd(x.data_ptr(), w.data_ptr(), dy.data_ptr(), rstd.data_ptr(),
                               dres.data_ptr() if dres is not None else None, dx.data_ptr(), dw.data_ptr(),
                               scratch.data_ptr(), T, D, 0, _lib.stream_ptr()), "gf_rmsnorm_bwd")
        return dx, dw
    xf, gf, wf = x.float(), dy.float(), w.float()
    g = gf * wf
    r = rstd[:, None]
    dx = r * g - xf * (r ** 3) * (g * xf).mean(-1, keepdim=True)
    if dres is not None:
        dx = dx + dres.float()
    dw = (gf * xf * r).sum(0)
    if dw_out is not None:
        dw_out.copy_(dw.to(dw_out.dtype))
        dw = dw_out
    else:
        dw = dw.to(w.dtype)
    return dx.to(x.dtype), dw


# ------------------------------------------------------------------ RoPE (in place on [T, H, D] views)
def rope_(x3, cos, sin, S, interleaved=False, pos_offset=0, backward=False):
    T, H, D = x3.shape
    if _k(x3):
        check_rope_tables(x3.device, S, D, cos, sin, pos_offset)
        _rc(_lib.cuda_lib().gf_rope(x3.data_ptr(), cos.data_ptr(), sin.data_ptr(), T, H, D, x3.stride(0),
                                    x3.stride(1), S, pos_offset, 1 if interleaved else 0, 1 if backward else 0,
                                    _lib.stream_ptr()), "gf_rope")
        return x3
    xb = x3.reshape(T // S, S, H, D)
    s = -sin if backward else sin
    x3.copy_(rope_ref(xb, cos, s, interleaved, pos_offset).reshape(T, H, D))
    return x3


# ------------------------------------------------------------------ SwiGLU
def swiglu_fwd(gu):
    T, F2 = gu.shape
    if _k(gu):
        y = torch.empty((T, F2 // 2), dtype=gu.dtype, device=gu.device)
        _rc(_lib.cuda_lib().gf_swiglu_fwd(gu.data_ptr(), y.data_ptr(), T, F2 // 2, _lib.stream_ptr()),
            "gf_swiglu_fwd")
        return y
    g, u = gu.float().chunk(2, -1)
    return (F.silu(g) * u).to(gu.dtype)


def swiglu_bwd(gu, dy, out=None):
    T, F2 = gu.shape
    if _k(gu):
        dgu = out if out is not None else torch.empty_like(gu)
        _rc(_lib.cuda_lib().gf_swiglu_bwd(gu.data_ptr(), dy.data_ptr(), dgu.data_ptr(), T, F2 // 2,
                                          _lib.stream_ptr()), "gf_swiglu_bwd")
        return dgu
    g, u = gu.float().chunk(2, -1)
    s = torch.sigmoid(g)
    d = dy.float()
    return torch.cat((d * u * (s + g * s * (1 - s)), d * g * s), -1).to(gu.dtype)


# ------------------------------------------------------------------ attention on packed rows
def attn_fwd(q, k, v, B, S, Hq, Hkv, D, causal=True, scale=None):
    """q: [B*S, Hq*D] view (row pitch free), k/v: [B*S, Hkv*D] views. Returns (o [B*S, Hq*D], lse [B,Hq,S])."""
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    if _k(q):
        o = torch.empty((B * S, Hq * D), dtype=q.dtype, device=q.device)
        lse = torch.empty((B, Hq, S), dtype=torch.float32, device=q.device)
        _rc(_lib.flash_fwd_fn()(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(),
                                              B, S, Hq, Hkv, D, q.stride(0), k.stride(0), v.stride(0), Hq * D,
                                              float(scale), 1 if causal else 0,
                                              _lib.status_word(q.device).data_ptr(), _lib.stream_ptr()),
            "gf_flash_attn_fwd")
        return o, lse
    qf = q.float().reshape(B, S, Hq, D).transpose(1, 2)
    kf = k.float().reshape(B, S, Hkv, D).transpose(1, 2).repeat_interleave(Hq // Hkv, 1)
    vf = v.float().reshape(B, S, Hkv, D).transpose(1, 2).repeat_interleave(Hq // Hkv, 1)
    s = qf @ kf.transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=q.device).tril(), float("-inf"))
    lse = torch.logsumexp(s, -1)
    o = (torch.softmax(s, -1) @ vf).transpose(1, 2).reshape(B * S, Hq * D).to(q.dtype)
    return o, lse


def attn_bwd(q, k, v, o, do, lse, dq, dk, dv, B, S, Hq, Hkv, D, causal=True, scale=None):
    """Writes dq/dk/dv (row-pitched views, e.g. slices of one packed dqkv buffer)."""
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    if _k(q):
        _lib.flash_attn_backward(q, k, v, o, do, lse, dq, dk, dv, B, S, Hq, Hkv, D,
                                 dict(q=q.stride(0), k=k.stride(0), v=v.stride(0), o=o.stride(0), do=do.stride(0),
                                      dq=dq.stride(0), dk=dk.stride(0), dv=dv.stride(0)), scale, causal)
        return
    G = Hq // Hkv
    qf = q.float().reshape(B, S, Hq, D).transpose(1, 2)
    kf = k.float().reshape(B, S, Hkv, D).transpose(1, 2).repeat_interleave(G, 1)
    vf = v.float().reshape(B, S, Hkv, D).transpose(1, 2).repeat_interleave(G, 1)
    dof = do.float().reshape(B, S, Hq, D).transpose(1, 2)
    s = qf @ kf.transpose(-1, -2) * scale
    if causal:
        s = s.masked_fill(~torch.ones(S, S, dtype=torch.bool, device=q.device).tril(), float("-inf"))
    # probabilities from the given log-sum-exp and delta from o, as in the kernel: k/v may be one block of a longer
    # key sequence (ring attention), in which case lse and o are those of the whole row
    p = torch.exp(s - lse.float().unsqueeze(-1))
    of = o.float().reshape(B, S, Hq, D).transpose(1, 2)
    dvf = p.transpose(-1, -2) @ dof
    dp = dof @ vf.transpose(-1, -2)
    ds = p * (dp - (dof * of).sum(-1, keepdim=True)) * scale
    dqf = ds @ kf
    dkf = ds.transpose(-1, -2) @ qf
    dkf = dkf.reshape(B, Hkv, G, S, D).sum(2)
    dvf = dvf.reshape(B, Hkv, G, S, D).sum(2)
    dq.copy_(dqf.transpose(1, 2).reshape(B * S, Hq * D).to(dq.dtype))
    dk.copy_(dkf.transpose(1, 2).reshape(B * S, Hkv * D).to(dk.dtype))
    dv.copy_(dvf.transpose(1, 2).reshape(B * S, Hkv * D).to(dv.dtype))


# ------------------------------------------------------------------ loss
def xent_fwd_bwd(logits, targets, grad_scale=None):
    """Mean cross-entropy; overwrites ``logits`` with d(loss)/d(logits). Returns the fp32 scalar loss tensor."""
    T, V = logits.shape
    scale = (1.0 / T) if grad_scale is None else grad_scale
    if _k(logits):
        loss_rows = torch.empty(T, dtype=torch.float32, device=logits.device)
        _rc(_lib.cuda_lib().gf_xent_fused(logits.data_ptr(), targets.data_ptr(), loss_rows.data_ptr(),
                                          logits.data_ptr(), T, V, logits.stride(0), float(scale), -(1 << 62),
                                          _lib.status_word(logits.device).data_ptr(), _lib.stream_ptr()),
            "gf_xent_fused")
        return loss_rows.sum() * scale
    lf = logits.float()
    lse = torch.logsumexp(lf, -1)
    loss_rows = lse - lf.gather(1, targets[:, None]).squeeze(1)
    p = torch.softmax(lf, -1)
    p[torch.arange(T), targets] -= 1.0
    logits.copy_((p * scale).to(logits.dtype))
    return loss_rows.sum() * scale


# ------------------------------------------------------------------ optimizer
def adamw_flat(p32, m, v, g, p_lp, *, lr, beta1, beta2, eps, weight_decay, step, grad_scale=1.0, decoupled=True):
    if p32.is_cuda:
        from .optim_kernels import adam_flat

        adam_flat(p32, m, v, g, p_lp, lr=lr, beta1=beta1, beta2=beta2, eps=eps, weight_decay=weight_decay,
                  step=step, grad_scale=grad_scale, decoupled=decoupled)
        return
    gf = g.float() * grad_scale
    if not decoupled:
        gf = gf + weight_decay * p32
    m.mul_(beta1).add_(gf, alpha=1 - beta1)
    v.mul_(beta2).addcmul_(gf, gf, value=1 - beta2)
    mh = m / (1 - beta1 ** step)
    vh = v / (1 - beta2 ** step)
    if decoupled:
        p32.mul_(1 - lr * weight_decay)
    p32.sub_(lr * mh / (vh.sqrt() + eps))
    if p_lp is not None:
        p_lp.copy_(p32.to(p_lp.dtype))


# ------------------------------------------------------------------ decode attention over a KV cache
# up to eight the merge reads all pieces at once; of more, only 16 was ever the best
_SLICES = 1, 2, 3, 4, 5, 6, 7, 8, 16


@functools.lru_cache(maxsize=1024)
def _even_slices(ctas: int, blocks: int, D: int, sms: int) -> int:
    """Slices of the cache for sequences of one length (``blocks`` of 128 rows, the shortest slice), ``ctas`` CTAs to a slice: the number
    with the least estimated time. That is a wave of CTAs after the other (two to an SM, four with D = 64), a full one at
    memory speed, the last one as long as its fullest SM needs: one, two, three CTAs of an SM take .53 and .72 of a full
    wave (D = 64: .32, .44, .58, then .93); as long as 85 rows for another wave, 70 for the merge, 3 for each slice in it, 70 for more
    than eight. Over 351 combinations of 1 to 64 sequences, 2 to 32 heads in the cache and 64 to 8000 keys the choice takes
    0.3 % longer than the best one on average and 9 % at most. Measured, us with 1 / 2 / 3 / 4 / 8 / 16 slices: D = 128, 8 CTAs at 4000 keys
    50.5 / 28.2 / 20.4 / 16.7 / 10.8 / 9.9; 160 CTAs at 4000 61.4 / 73.9 / 54.7 / 63.0 / 58.8; 248 CTAs at 4000 79.9 / 80.9 / 85.0 / 88.7 / 88.6; 96 CTAs at 300, 1 / 2
    6.8 / 7.6; D = 64, 32 CTAs at 2048 18.0 / 12.0 / 9.7 / 8.5 / 7.9 / 10.8; 256 CTAs at 4000 42.9 / 47.6 / 52.8 / 46.9 / 48.6."""
    steps = (.53, .72) if D > 64 else (.32, .44, .58, .93)
    slots, n = sms * len(steps), 128 * blocks
    best = cost = None
    for s in _SLICES:
        if s > max(1, blocks):
            break
        waves, rest = divmod(ctas * s, slots)
        tail = max(steps[-(-rest // sms) - 1], rest / slots) if rest else 0.
        c = -(-n // s) * (waves + tail) + 85 * (waves - (not rest)) + (70 + 3 * s + 70 * (s > 8) if s > 1 else 0)
        if best is None or c < cost:
            best, cost = s, c
    return best


@functools.lru_cache(maxsize=1024)
def _decode_parts(B: int, Hkv: int, n: int, D: int, sms: int, per_seq: bool) -> int:
    """How decode attention cuts the keys of ``B`` sequences of at most ``n`` keys: parts of each sequence, or, negative, the number of
    parts of all sequences together (one wave of CTAs, whatever the lengths are).

    Lengths that differ are not known here. Slices of each sequence: a piece takes .34 of a full wave's time (D = 64: .2) and up to .15 more
    as the machine fills, a wave of CTAs more as long as 150 rows, the merge 52, each slice in it 6, more than eight 110. Shares
    of all sequences cost 5 us for finding a share's sequences and the pieces that begin and end inside one, and are taken where there
    are 40 units of 64 keys to a CTA and sequences of 2048 keys: lengths far apart then matter more. Over 219 combinations of 2 to
    64 sequences and 130 to 8000 keys, with lengths uniform / one in eight long and the others a 16th / all full, the choice takes 3 /
    6 / 6 % longer than the best of all on average. us with 1 / 2 / 4 / 8 slices / shares, uniform lengths: 62 sequences of 1 .. 300, 64 /
    8 heads of 128 15.6 / 25.8 / 33.2 / - / 28.2; 4 of 1 .. 4000, 64 / 8 heads of 128 39.1 / 23.8 / 15.7 / 13.0 / 16.5; 8 of 1 .. 4000, 32 / 8 heads
    of 64 24.4 / 15.5 / 12.2 / 11.0 / 14.2; 32 of 1 .. 4000, 32 / 8 heads of 128 62.1 / 59.9 / 53.8 / 57.1 / 54.8, one in eight long
    55.6 / 41.7 / 34.9 / 31.2 / 28.8."""
    heads = max(1, B * Hkv)
    if not per_seq:
        return _even_slices(heads, max(1, (n + 127) // 128), D, sms)
    slots, units = sms * (2 if D > 64 else 4), (n + 63) // 64
    if units >= 32 and heads * units >= 40 * slots:
        return -max(1, slots // Hkv)
    piece = .34 if D > 64 else .2
    cost = lambda s: (64 * -(-units // s) * (piece + .15 * min(1., heads * s / slots))  # noqa: E731
                      + 150 * max(0., heads * s / slots - 1) + (52 + 6 * s + 110 * (s > 8) if s > 1 else 0))
    return min((s for s in _SLICES if s <= max(1, units)), key=cost)


def attn_decode(q, kcache, vcache, length, B, Hq, Hkv, D, scale=None, splits=None, out=None):
    """q [B, Hq * D]; caches [B, s_max, Hkv * D]; attends over the first ``length`` cache rows of every sequence
    (``length``: int, or an int32 tensor [B] of per-sequence lengths). Returns [B, Hq * D]."""
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    if _k(q):
        s_max = kcache.shape[1]
        per_seq = torch.is_tensor(length)
        n = s_max if per_seq else int(length)
        if splits is None:
            splits = _decode_parts(B, Hkv, n, D, _sm_count(q.device), per_seq)
        elif splits < 1:
            raise ValueError(f"attn_decode cuts the keys of a head into one part or more, not {splits}")
        if out is None:
            out = torch.empty(B, Hq * D, dtype=q.dtype, device=q.device)
        scratch = torch.empty((B * splits if splits > 0 else -2 * splits) * Hq * (D + 2), dtype=torch.float32, device=q.device)
        _rc(_lib.cuda_lib().gf_attn_decode(q.data_ptr(), q.stride(0), kcache.data_ptr(), vcache.data_ptr(), s_max,
                                           length.data_ptr() if per_seq else None, 0 if per_seq else n, out.data_ptr(),
                                           out.stride(0), B, Hq, Hkv, D, float(scale), splits, scratch.data_ptr(),
                                           _lib.stream_ptr()), "gf_attn_decode")
        return out
    G = Hq // Hkv
    res = torch.empty(B, Hq * D, dtype=q.dtype, device=q.device)
    for b in range(B):
        n = int(length[b]) if torch.is_tensor(length) else int(length)
        qf = q[b].float().view(Hkv, G, D)
        kf = kcache[b, :n].float().view(n, Hkv, D).permute(1, 0, 2)
        vf = vcache[b, :n].float().view(n, Hkv, D).permute(1, 0, 2)
        p = torch.softmax(qf @ kf.transpose(-1, -2) * scale, -1)
        res[b] = (p @ vf).reshape(Hq * D).to(q.dtype)
    if out is not None:
        out.copy_(res)
        return out
    return res


# ------------------------------------------------------------------ one decoder layer, one token of each sequence
def llama_decode_layer(x, attn_norm, attn_eps, wqkv, wo, ffn_norm, ffn_eps, gate_up, down, cos, sin, kcache, vcache, Hq, Hkv, D,
                       interleaved, pos):
    """A whole LLaMA decoder layer for one new token of each of at most 64 sequences, in one call of the kernel library (seven kernels
    or nine, most of them started while the one in front of them ends). ``x [B, hidden]`` or ``[B, 1, hidden]`` and weights ``[out, in]``
    dense bf16; caches ``[B, s_max, Hkv, D]`` dense, row ``pos`` is written; tables fp32 with a row for ``pos``. Returns the shape of ``x``."""
    B, hidden = x.shape[0], x.shape[-1]
    inner, s_max = down.shape[1], kcache.shape[1]
    splits = _even_slices(B * Hkv, (pos + 128) // 128, D, _sm_count(x.device))
    lib = _lib.cuda_lib()
    y = torch.empty_like(x)
    # workspaces of the layer: q, k, v; attention; its sum with x; gate and up; the parts of the attention (fp32)
    ws = torch.empty(2 * B * ((2 * Hq + 2 * Hkv) * D + hidden + 2 * inner + max(hidden, inner))
                     + 4 * B * Hq * splits * (D + 2) + 1536, dtype=torch.uint8, device=x.device)
    _rc(lib.gf_llama_decode_layer(
        x.data_ptr(), attn_norm.data_ptr(), float(attn_eps), wqkv.data_ptr(), wo.data_ptr(), ffn_norm.data_ptr(),
        float(ffn_eps), gate_up.data_ptr(), down.data_ptr(), cos.data_ptr(), sin.data_ptr(), kcache.data_ptr(),
        vcache.data_ptr(), s_max, y.data_ptr(), ws.data_ptr(), B, hidden, inner, Hq, Hkv, D, 1 if interleaved else 0, pos, splits,
        _lib.status_word(x.device).data_ptr(), _lib.stream_ptr()), "gf_llama_decode_layer")
    if _lib.DEBUG_SYNC:
        _lib.check_status(x.device)
    return y


def rmsnorm_gemm(x, norm_w, eps, w):
    """``rms_norm(x) @ w^T`` for at most 16 rows of dense bf16, in one kernel (the norm in front of the product). ``w [N, K]`` dense; rows
    of the result start on 16-byte boundaries."""
    (M, K), N = x.shape, w.shape[0]
    bf16, dev = torch.bfloat16, x.device
    if not (norm_w.shape == (K,) and w.shape == (N, K) and x.dtype is bf16 and norm_w.dtype is bf16 and w.dtype is bf16
            and norm_w.device == dev and w.device == dev and x.is_contiguous() and norm_w.is_contiguous() and w.is_contiguous()):
        raise ValueError(f"rmsnorm_gemm takes dense bf16 tensors [M, K], [K], [N, K] on one device, not {list(x.shape)}, "
                         f"{list(norm_w.shape)}, {list(w.shape)}")
    y = torch.empty((M, N if N % 8 == 0 else (N + 63) // 64 * 64), dtype=x.dtype, device=x.device)[:, :N]
    _rc(_lib.cuda_lib().gf_gemm_rows(x.data_ptr(), K, w.data_ptr(), K, y.data_ptr(), y.stride(0), 0, M, N, K, 1, norm_w.data_ptr(),
                                     float(eps), None, None, 0, 1.0, 0, _lib.status_word(x.device).data_ptr(), _lib.stream_ptr()),
        "gf_gemm_rows")
    if _lib.DEBUG_SYNC:
        _lib.check_status(x.device)
    return y
