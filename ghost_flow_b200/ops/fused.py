"""Autograd functions over the hand-written sm_100a kernels: RMSNorm, LayerNorm, RoPE, SwiGLU,
GELU-family activations, softmax cross-entropy and FlashAttention.

Every function takes the CUDA path for bf16 CUDA tensors and a plain PyTorch fp32-capable path for
CPU tensors (used by the CPU configuration and the CPU test-suite). The PyTorch path is also the
numerical reference the GPU tests compare against.
"""
from __future__ import annotations

import ctypes
import functools
import math
import os

import torch
import torch.nn.functional as F
from torch.autograd import forward_ad
from torch.utils._device import DeviceContext

from . import _lib

def _scratch(device, nfloats: int) -> torch.Tensor:
    """fp32 workspace of one call (partial sums of the norm backward kernels). From torch's allocator, so that it belongs to
    the current stream, or to the graph's pool while a CUDA graph is recorded: one buffer kept for all calls would be
    shared by streams, and a recorded graph would go on writing it after it was replaced by a larger one."""
    return torch.empty(nfloats, dtype=torch.float32, device=device)


def _cuda_bf16(*ts) -> bool:
    return all(t is None or (t.is_cuda and t.dtype == torch.bfloat16) for t in ts)


class _NoGraph:
    """Stand-in for the autograd context when nothing needs a gradient: the forward of an autograd function is then
    called directly, which skips the cost of creating a graph node (several microseconds per call on the host)."""

    needs_input_grad = ()

    def save_for_backward(self, *tensors):
        pass

    def mark_dirty(self, *tensors):
        pass


def _call(fn, *args):
    """``fn.apply(*args)`` when a gradient may be wanted, else ``fn.forward`` without a graph node."""
    if torch.is_grad_enabled():
        for a in args:
            if isinstance(a, torch.Tensor) and a.requires_grad:
                return fn.apply(*args)
    return fn.forward(_NoGraph(), *args)


def _rc(rc, what):
    _lib.check_rc(rc, what)
    if _lib.DEBUG_SYNC:
        _lib.check_status()


# ------------------------------------------------------------------------------------------ RMSNorm
def _dense(t):
    return t if t.is_contiguous() else t.contiguous()


class _RMSNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, eps, residual):
        D = x.shape[-1]
        x_is_leaf = x.is_leaf
        x = _dense(x)
        T = x.numel() // D
        y = torch.empty_like(x)
        # the row statistics are kept for the backward pass only
        rstd = torch.empty(T, dtype=torch.float32, device=x.device) if type(ctx) is not _NoGraph else None
        h = res = None
        if residual is not None:
            res = _dense(residual)
            h = torch.empty_like(x)
        _rc(_lib.cuda_lib().gf_rmsnorm_fwd(
            x.data_ptr(), None if res is None else res.data_ptr(), w.data_ptr(), y.data_ptr(),
            None if h is None else h.data_ptr(), None if rstd is None else rstd.data_ptr(), T, D, float(eps),
            _lib.stream_ptr()), "gf_rmsnorm_fwd")
        ctx.save_for_backward(h if h is not None else x, w, rstd)
        ctx.has_res = residual is not None
        # A call on two leaves only (inside a model both are results of other modules): they keep their gradients apart, so the kernel
        # writes both, where autograd would copy one (a pass of its own).
        ctx.two = residual is not None and x_is_leaf and residual.is_leaf
        return (y, h) if residual is not None else y

    @staticmethod
    def backward(ctx, dy, dh=None):
        x, w, rstd = ctx.saved_tensors
        D = x.shape[-1]
        T = x.numel() // D
        dy = _dense(dy)
        dres = _dense(dh) if (ctx.has_res and dh is not None) else None
        dx = torch.empty_like(x)
        dx2 = torch.empty_like(x) if ctx.two and ctx.needs_input_grad[0] and ctx.needs_input_grad[3] else None
        dw = torch.empty_like(w)
        lib = _lib.cuda_lib()
        g = lib.gf_norm_bwd_grid(T)
        scratch = _scratch(x.device, g * D)
        _rc(lib.gf_rmsnorm_bwd2(x.data_ptr(), w.data_ptr(), dy.data_ptr(), rstd.data_ptr(),
                                None if dres is None else dres.data_ptr(), dx.data_ptr(),
                                None if dx2 is None else dx2.data_ptr(), dw.data_ptr(), scratch.data_ptr(), T, D, 0,
                                _lib.stream_ptr()), "gf_rmsnorm_bwd2")
        return dx, dw, None, None if not ctx.has_res else dx if dx2 is None else dx2


def rms_norm_ref(x, w, eps=1e-6):
    xf = x.float()
    y = xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps) * w.float()
    return y.to(x.dtype)


def rms_norm(x, w, eps: float = 1e-6, residual=None):
    """RMSNorm; with ``residual`` returns ``(norm(x + residual), x + residual)`` from one kernel."""
    if _cuda_bf16(x, w, residual):
        return _call(_RMSNormFn, x, w, eps, residual)
    if residual is not None:
        h = x + residual
        return rms_norm_ref(h, w, eps), h
    return rms_norm_ref(x, w, eps)


# ------------------------------------------------------------------------------------------ LayerNorm
class _LayerNormFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, b, eps):
        D = x.shape[-1]
        x = _dense(x)
        T = x.numel() // D
        y = torch.empty_like(x)
        stats = torch.empty((2, T), dtype=torch.float32, device=x.device) if type(ctx) is not _NoGraph else None
        lib = _lib.cuda_lib()
        _rc(lib.gf_layernorm_fwd(x.data_ptr(), w.data_ptr(), b.data_ptr() if b is not None else None, y.data_ptr(),
                                 None if stats is None else stats.data_ptr(),
                                 None if stats is None else stats.data_ptr() + 4 * T, T, D, float(eps),
                                 _lib.stream_ptr()), "gf_layernorm_fwd")
        ctx.save_for_backward(x, w, stats)
        ctx.has_bias = b is not None
        return y

    @staticmethod
    def backward(ctx, dy):
        x, w, stats = ctx.saved_tensors
        D = x.shape[-1]
        T = x.numel() // D
        dy = _dense(dy)
        dx = torch.empty_like(x)
        dw = torch.empty_like(w)
        db = torch.empty_like(w) if ctx.has_bias else None
        lib = _lib.cuda_lib()
        g = lib.gf_norm_bwd_grid(T)
        scratch = _scratch(x.device, 2 * g * D)
        _rc(lib.gf_layernorm_bwd(x.data_ptr(), w.data_ptr(), dy.data_ptr(), stats.data_ptr(), stats.data_ptr() + 4 * T,
                                 dx.data_ptr(), dw.data_ptr(), db.data_ptr() if db is not None else None,
                                 scratch.data_ptr(), T, D, 0, _lib.stream_ptr()), "gf_layernorm_bwd")
        return dx, dw, db, None


def layer_norm(x, w, b=None, eps: float = 1e-5):
    if _cuda_bf16(x, w, b) and x.shape[-1] % 8 == 0 and x.shape[-1] <= 8192:
        return _call(_LayerNormFn, x, w, b, eps)
    return F.layer_norm(x, (x.shape[-1],), w, b, eps)


# ------------------------------------------------------------------------------------------ RoPE
_ROPE_CACHE = {}


def rope_tables(seq_len: int, head_dim: int, theta: float = 10000.0, device="cpu"):
    """fp32 cos/sin tables ``[seq_len, head_dim/2]`` (angle = pos * theta^(-2i/d))."""
    key = (seq_len, head_dim, float(theta), str(device))
    t = _ROPE_CACHE.get(key)
    if t is None:
        inv = 1.0 / (theta ** (torch.arange(0, head_dim, 2, dtype=torch.float64) / head_dim))
        ang = torch.outer(torch.arange(seq_len, dtype=torch.float64), inv)
        t = (ang.cos().float().to(device).contiguous(), ang.sin().float().to(device).contiguous())
        _ROPE_CACHE[key] = t
    return t


def rope_ref(x, cos, sin, interleaved=False, pos_offset=0):
    """x: [..., S, H, D]; cos/sin: [>=S+pos_offset, D/2]."""
    S = x.shape[-3]
    c = cos[pos_offset:pos_offset + S].unsqueeze(-2).to(torch.float32)
    s = sin[pos_offset:pos_offset + S].unsqueeze(-2).to(torch.float32)
    xf = x.float()
    if interleaved:
        a, b = xf[..., 0::2], xf[..., 1::2]
        out = torch.stack((a * c - b * s, b * c + a * s), dim=-1).flatten(-2)
    else:
        h = x.shape[-1] // 2
        a, b = xf[..., :h], xf[..., h:]
        out = torch.cat((a * c - b * s, b * c + a * s), dim=-1)
    return out.to(x.dtype)


def check_rope_tables(device, S: int, D: int, cos, sin, pos_offset: int) -> None:
    """Raises where the kernels, which index the tables by position without a bound, would read outside of them."""
    c = cos.shape
    if c == sin.shape and len(c) == 2 and 2 * c[1] == D and 0 <= pos_offset <= c[0] - S and cos.device == sin.device == device:
        return
    if not (cos.device == sin.device == device and cos.dim() == sin.dim() == 2 and cos.shape[1] == sin.shape[1] == D // 2):
        raise ValueError(f"rope tables must be [positions, {D // 2}] on {device}, got {list(cos.shape)} on {cos.device} "
                         f"and {list(sin.shape)} on {sin.device}")
    if pos_offset < 0 or pos_offset + S > min(cos.shape[0], sin.shape[0]):
        raise ValueError(f"rope positions {pos_offset} .. {pos_offset + S - 1} are not in tables of "
                         f"{min(cos.shape[0], sin.shape[0])} rows")


def _rope_tables_fit_kernel(cos, sin) -> bool:
    return (cos.dtype == torch.float32 and sin.dtype == torch.float32 and cos.is_contiguous() and sin.is_contiguous()
            and cos.data_ptr() % 16 == 0 and sin.data_ptr() % 16 == 0)


def _rope_launch(x, cos, sin, S, interleaved, pos_offset, backward):
    """In place on x viewed as [T, H, D] (unit stride over D; rows and heads may be strided)."""
    T, H, D = x.shape
    lib = _lib.cuda_lib()
    _rc(lib.gf_rope(x.data_ptr(), cos.data_ptr(), sin.data_ptr(), T, H, D, x.stride(0), x.stride(1), S, pos_offset,
                    1 if interleaved else 0, 1 if backward else 0, _lib.stream_ptr()), "gf_rope")


class _RopeFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, cos, sin, interleaved, pos_offset, inplace):
        # x: [B, S, H, D] (any row/head strides)
        B, S, H, D = x.shape
        out = x if inplace else x.clone()
        v = out.view(B * S, H, D) if out.is_contiguous() else out.reshape(B * S, H, D)
        if v.data_ptr() != out.data_ptr() or v.stride(2) != 1:
            raise RuntimeError("rope needs a [B,S,H,D] tensor whose (B,S) dims can be flattened without a copy")
        _rope_launch(v, cos, sin, S, interleaved, pos_offset, False)
        ctx.save_for_backward(cos, sin)
        ctx.args = (S, interleaved, pos_offset)
        if inplace:
            ctx.mark_dirty(x)
        return out

    @staticmethod
    def backward(ctx, dy):
        cos, sin = ctx.saved_tensors
        S, interleaved, pos_offset = ctx.args
        g = dy.contiguous().clone()
        B, S_, H, D = g.shape
        _rope_launch(g.view(B * S_, H, D), cos, sin, S, interleaved, pos_offset, True)
        return g, None, None, None, None, None


def rope(x, cos, sin, interleaved: bool = False, pos_offset: int = 0, inplace: bool = False):
    """Rotary embedding on ``[B, S, H, D]``; half-split pairing by default, ``interleaved`` for (2i, 2i+1)."""
    if x.is_cuda and x.dtype == torch.bfloat16 and x.shape[-1] % 16 == 0:
        check_rope_tables(x.device, x.shape[-3], x.shape[-1], cos, sin, pos_offset)
        if _rope_tables_fit_kernel(cos, sin):
            return _call(_RopeFn, x, cos, sin, interleaved, pos_offset, inplace)
    return rope_ref(x, cos, sin, interleaved, pos_offset)


def _packed_rows(t):
    """``t [B, S, H, D]`` as it is when its rows can be addressed as ``base + (b * S + s) * pitch`` on 16-byte boundaries
    with the heads packed, else a contiguous copy; with the row pitch."""
    ld = _rows_view(t)
    if ld is None or ld % 8 or t.data_ptr() % 16:
        t = t.clone(memory_format=torch.contiguous_format)
        ld = t.shape[2] * t.shape[3]
    return t, ld


def _rope_qkv_launch(src, dst, B, S, H, Hk, D, cos, sin, interleaved, pos_offset, backward):
    """Rotates q and k and copies v. ``src``: (address, row pitch) of each, heads packed; ``dst``: (address, row pitch,
    sequence pitch) of each, v's ``None`` to leave it alone."""
    (q, ldq), (k, ldk), (v, ldv) = src
    qd, kd, vd = dst
    table = (ctypes.c_longlong * 9)(ldq, ldk, ldv, qd[1], qd[2], kd[1], kd[2], *((0, 0) if vd is None else vd[1:]))
    _rc(_lib.cuda_lib().gf_rope_qkv(q, k, v, qd[0], kd[0], None if vd is None else vd[0], table, cos.data_ptr(),
                                    sin.data_ptr(), B * S, S, H, Hk, D, pos_offset, 1 if interleaved else 0,
                                    1 if backward else 0, _lib.stream_ptr()), "gf_rope_qkv")


def _packed_qkv(qkv, H: int, Hk: int):
    """q, k and v of a packed projection as sources of :func:`_rope_qkv_launch`, and the tensor they point into."""
    t, ld = _packed_rows(qkv)
    p, head = t.data_ptr(), 2 * t.shape[3]
    return t, ((p, ld), (p + H * head, ld), (p + (H + Hk) * head, ld))


class _RopeQKVFn(torch.autograd.Function):
    """Split and rotation of a packed projection in one launch per direction: the backward pass rotates the gradients of
    q and k back and packs the three gradients in the same pass."""

    @staticmethod
    def forward(ctx, qkv, H, Hk, cos, sin, interleaved, pos_offset):
        B, S, G, D = qkv.shape
        q = torch.empty((B, S, H, D), dtype=qkv.dtype, device=qkv.device)
        k = torch.empty((B, S, Hk, D), dtype=qkv.dtype, device=qkv.device)
        v = qkv[:, :, H + Hk:]
        t, src = _packed_qkv(qkv, H, Hk)
        _rope_qkv_launch(src, ((q.data_ptr(), H * D, S * H * D), (k.data_ptr(), Hk * D, S * Hk * D), None), B, S, H, Hk, D,
                         cos, sin, interleaved, pos_offset, False)
        ctx.save_for_backward(cos, sin)
        ctx.args = (H, Hk, interleaved, pos_offset)
        return q, k, v

    @staticmethod
    def backward(ctx, dq, dk, dv):
        cos, sin = ctx.saved_tensors
        H, Hk, interleaved, pos_offset = ctx.args
        B, S, _, D = dq.shape
        G = H + 2 * Hk
        g = torch.empty((B, S, G, D), dtype=dq.dtype, device=dq.device)
        p = g.data_ptr()
        packed = [_packed_rows(t) for t in (dq, dk, dv)]
        _rope_qkv_launch([(t.data_ptr(), ld) for t, ld in packed],
                         [(p + 2 * h * D, G * D, S * G * D) for h in (0, H, H + Hk)], B, S, H, Hk, D, cos, sin, interleaved,
                         pos_offset, True)
        return g, None, None, None, None, None, None


def _rope_qkv_ok(qkv, H, Hk, cos, sin, pos_offset) -> bool:
    if qkv.shape[2] != H + 2 * Hk:
        raise ValueError(f"a packed projection of {H} + 2 x {Hk} heads has {H + 2 * Hk} of them, not {qkv.shape[2]}")
    if not (qkv.is_cuda and qkv.dtype == torch.bfloat16 and qkv.shape[-1] % 16 == 0 and qkv.numel() > 0):
        return False
    check_rope_tables(qkv.device, qkv.shape[1], qkv.shape[3], cos, sin, pos_offset)
    return _rope_tables_fit_kernel(cos, sin)


def rope_qkv(qkv, num_heads: int, num_kv_heads: int, cos, sin, interleaved: bool = False, pos_offset: int = 0):
    """``q, k, v`` of a packed projection output ``[B, S, H + 2 Hk, D]`` with q and k rotated (see :func:`rope`)."""
    H, Hk = num_heads, num_kv_heads
    if _rope_qkv_ok(qkv, H, Hk, cos, sin, pos_offset):
        return _call(_RopeQKVFn, qkv, H, Hk, cos, sin, interleaved, pos_offset)
    q, k, v = split_qkv(qkv, H, Hk)
    return rope(q, cos, sin, interleaved, pos_offset), rope(k, cos, sin, interleaved, pos_offset), v


def _rows_apart(row: int, dims) -> bool:
    """Whether rows of ``row`` elements repeated over ``dims`` = (stride, count) pairs share no element (sufficient: every
    stride reaches over all that lies inside it)."""
    extent = row
    for st, n in sorted(dims):
        if n > 1:
            if st < extent:
                return False
            extent += st * (n - 1)
    return True


def _cache_rows_apart(kc, vc) -> bool:
    """Whether no two rows of the caches ``[B, n, Hk, D]`` (packed heads) share memory: expanded caches are refused by the
    assignments, and two that overlap are written by them one after the other."""
    (B, n, Hk, D), sk, sv = kc.shape, kc.stride(), vc.stride()
    row, between = Hk * D, abs(kc.data_ptr() - vc.data_ptr()) // kc.element_size()
    if sk == sv and sk[1] == row and sk[0] == n * row:        # two dense caches
        return between >= B * sk[0]
    dims = [(sk[0], B), (sk[1], n)], [(sv[0], B), (sv[1], n)]
    if sk[:2] == sv[:2]:                 # the caches themselves are one more dimension, wherever it lies
        return _rows_apart(row, [*dims[0], (between, 2)])
    ends = sorted((c.data_ptr(), c.data_ptr() + c.element_size() * (row + sum(st * (n - 1) for st, n in d)))
                  for c, d in zip((kc, vc), dims))
    return all(_rows_apart(row, d) for d in dims) and ends[0][1] <= ends[1][0]


def _cache_fits_kernel(c, shape, device, dtype) -> bool:
    s = c.stride()
    return (c.shape == shape and s[3] == 1 and s[2] == shape[3] and not (s[0] | s[1]) & 7 and not c.data_ptr() & 15
            and c.dtype is dtype and c.device == device)


def rope_qkv_to_cache(qkv, num_heads: int, num_kv_heads: int, cos, sin, kcache, vcache, interleaved: bool = False,
                      pos_offset: int = 0):
    """Rotated q of a packed projection output; rotated k and v go to rows ``pos_offset ..`` of the caches
    ``[B, max_len, Hk, D]``. Inference only: nothing is recorded for autograd."""
    B, S, _, D = qkv.shape
    H, Hk, n, dtype, device = num_heads, num_kv_heads, kcache.shape[1], qkv.dtype, qkv.device
    shape = (B, n, Hk, D)
    # what follows the assignments below (dispatch modes, transforms) would not see the kernel's writes
    if not torch.is_grad_enabled() and not _observed() and _rope_qkv_ok(qkv, H, Hk, cos, sin, pos_offset) \
            and pos_offset + S <= n and _cache_fits_kernel(kcache, shape, device, dtype) \
            and _cache_fits_kernel(vcache, shape, device, dtype) and _cache_rows_apart(kcache, vcache):
        q = torch.empty((B, S, H, D), dtype=dtype, device=device)
        t, src = _packed_qkv(qkv, H, Hk)
        at = [(c.data_ptr() + 2 * pos_offset * s1, s1, s0) for c in (kcache, vcache) for s0, s1, _, _ in (c.stride(),)]
        _rope_qkv_launch(src, ((q.data_ptr(), H * D, S * H * D), *at), B, S, H, Hk, D, cos, sin, interleaved, pos_offset, False)
        torch.autograd.graph.increment_version((kcache, vcache))     # a graph that saved a cache has to notice the write
        return q
    q, k, v = rope_qkv(qkv, H, Hk, cos, sin, interleaved, pos_offset)
    kcache[:, pos_offset:pos_offset + S] = k
    vcache[:, pos_offset:pos_offset + S] = v
    return q


# ------------------------------------------------------------------------------------------ SwiGLU / unary
class _SwiGLUFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, gu):
        F2 = gu.shape[-1]
        g2 = gu.reshape(-1, F2).contiguous()
        T = g2.shape[0]
        y = torch.empty((T, F2 // 2), dtype=gu.dtype, device=gu.device)
        _rc(_lib.cuda_lib().gf_swiglu_fwd(g2.data_ptr(), y.data_ptr(), T, F2 // 2, _lib.stream_ptr()),
            "gf_swiglu_fwd")
        ctx.save_for_backward(g2)
        ctx.shape = gu.shape
        return y.view(*gu.shape[:-1], F2 // 2)

    @staticmethod
    def backward(ctx, dy):
        (g2,) = ctx.saved_tensors
        T, F2 = g2.shape
        dy2 = dy.reshape(T, F2 // 2).contiguous()
        dgu = torch.empty_like(g2)
        _rc(_lib.cuda_lib().gf_swiglu_bwd(g2.data_ptr(), dy2.data_ptr(), dgu.data_ptr(), T, F2 // 2,
                                          _lib.stream_ptr()), "gf_swiglu_bwd")
        return dgu.view(ctx.shape)


def swiglu(gu):
    """``silu(gate) * up`` where ``gu = [..., gate | up]`` is the fused gate/up projection output."""
    if _cuda_bf16(gu) and (gu.shape[-1] // 2) % 8 == 0:
        return _call(_SwiGLUFn, gu)
    g, u = gu.chunk(2, dim=-1)
    return F.silu(g) * u


# private names of torch (tracing, torch.func transforms, dispatch modes, function modes, forward-mode level); a torch build
# without one of them counts as observed throughout, and the tensor-library form is taken
_PROBES = tuple(getattr(torch._C, n, None) for n in ("_get_tracing_state", "_are_functorch_transforms_active",
                                                      "_len_torch_dispatch_stack", "_len_torch_function_stack"))


_FUNCTION_MODES = getattr(torch.overrides, "_get_current_function_mode_stack", None)


def _only_device_contexts() -> bool:
    """Whether every function mode is a ``with torch.device(...)`` or ``torch.set_default_device``: they say where new tensors
    go, and follow nothing. Allocations next to a launch name their device."""
    return _FUNCTION_MODES is not None and all(type(m) is DeviceContext for m in _FUNCTION_MODES())


def _observed() -> bool:
    """Whether something follows the tensor operations of this call that a kernel launch would escape: tracing, compilation,
    ``torch.func`` transforms, dispatch or function modes, forward-mode gradients."""
    if None in _PROBES:
        return True
    tracing, transforms, dispatch_modes, function_modes = _PROBES
    return (tracing() is not None or transforms() or dispatch_modes() > 0
            or (function_modes() > 0 and not _only_device_contexts())
            or getattr(forward_ad, "_current_level", 0) >= 0 or torch.compiler.is_compiling())


observed = _observed


def decode_cache_ok(kcache, vcache, cos, sin, heads, device, pos: int) -> bool:
    """Whether a decoding kernel may write row ``pos`` of the caches ``[B, n, Hk, D]`` (``heads`` = B, Hk, D) and rotate with these
    tables; positions that are not in the tables are an error. For calls that nothing follows (:func:`observed`)."""
    B, Hk, D = heads
    if kcache.dim() != 4 or not (kcache.is_contiguous() and vcache.is_contiguous()):
        return False
    shape = (B, kcache.shape[1], Hk, D)
    if not (0 <= pos < shape[1] and _cache_fits_kernel(kcache, shape, device, torch.bfloat16)
            and _cache_fits_kernel(vcache, shape, device, torch.bfloat16) and _cache_rows_apart(kcache, vcache)):
        return False
    check_rope_tables(device, 1, D, cos, sin, pos)
    return _rope_tables_fit_kernel(cos, sin)


def embedding_rows(ids, table, rows: int | None = None):
    """``table[ids]`` with zero rows for ids outside the table, in one launch; ``None`` where the kernel does not apply
    (CPU tensors, a GPU that is not the current one, a gradient to record, rows that are no whole 16-byte vectors, tensors
    that are traced or transformed, a table of other than ``rows`` rows)."""
    if type(ids) is not torch.Tensor or type(table) not in (torch.Tensor, torch.nn.Parameter) or not table.is_cuda \
            or (torch.is_grad_enabled() and table.requires_grad) or _observed():
        return None
    if not (ids.is_cuda and ids.device == table.device and table.dim() == 2 and ids.numel() > 0
            and ids.dtype in (torch.int64, torch.int32) and table.dtype in (torch.bfloat16, torch.float32, torch.float16)
            and table.device.index == torch.cuda.current_device()     # launches go to the current device
            and table.is_contiguous() and table.shape[0] > 0 and rows in (None, table.shape[0])):
        return None
    row_bytes = table.shape[1] * table.element_size()
    if row_bytes == 0 or row_bytes % 16 or table.data_ptr() % 16:
        return None
    ids = _dense(ids)
    out = table.new_empty((*ids.shape, table.shape[1]))
    _rc(_lib.cuda_lib().gf_embedding_rows(ids.data_ptr(), 1 if ids.dtype is torch.int64 else 0, table.data_ptr(),
                                          out.data_ptr(), ids.numel(), table.shape[0], row_bytes, _lib.stream_ptr()),
        "gf_embedding_rows")
    return out


OPS = {"relu": 0, "gelu": 1, "sigmoid": 2, "tanh": 3, "silu": 4}


class _UnaryFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, op):
        xc = x.contiguous()
        y = torch.empty_like(xc)
        _rc(_lib.cuda_lib().gf_unary_fwd(xc.data_ptr(), y.data_ptr(), xc.numel(), op, 1, _lib.stream_ptr()),
            "gf_unary_fwd")
        ctx.save_for_backward(xc)
        ctx.op = op
        return y

    @staticmethod
    def backward(ctx, dy):
        (xc,) = ctx.saved_tensors
        dyc = dy.contiguous()
        dx = torch.empty_like(xc)
        _rc(_lib.cuda_lib().gf_unary_bwd_bf16(xc.data_ptr(), dyc.data_ptr(), dx.data_ptr(), xc.numel(), ctx.op,
                                              _lib.stream_ptr()), "gf_unary_bwd_bf16")
        return dx, None


def _unary_ref(x, name):
    if name == "relu":
        return torch.relu(x)
    if name == "gelu":
        return F.gelu(x, approximate="tanh")
    if name == "sigmoid":
        return torch.sigmoid(x)
    if name == "tanh":
        return torch.tanh(x)
    return F.silu(x)


def unary(x, name: str):
    """relu / gelu (tanh form) / sigmoid / tanh / silu."""
    if _cuda_bf16(x) and x.numel() % 8 == 0 and x.numel() > 0:
        return _call(_UnaryFn, x, OPS[name])
    return _unary_ref(x, name)


def gelu(x):
    return unary(x, "gelu")


def op_chain(x, names):
    """Applies a chain of unary ops in one pass over memory (inference helper, no autograd)."""
    if x.is_cuda and x.dtype in (torch.bfloat16, torch.float32) and len(names) <= 8:
        import ctypes

        xc = x.contiguous()
        y = torch.empty_like(xc)
        arr = (ctypes.c_int * len(names))(*[OPS[n] for n in names])
        _rc(_lib.cuda_lib().gf_op_chain(xc.data_ptr(), y.data_ptr(), xc.numel(), arr, len(names),
                                        1 if x.dtype == torch.bfloat16 else 0, _lib.stream_ptr()), "gf_op_chain")
        return y
    for n in names:
        x = _unary_ref(x, n)
    return x


# ------------------------------------------------------------------------------------------ cross-entropy
def _padded_rows(rows: int, cols: int, device, dtype, pitch: int | None = None) -> torch.Tensor:
    """``[rows, cols]`` view of a buffer whose row pitch is a multiple of 64 elements: every row starts on a 16-byte
    boundary whatever ``cols`` is (a 50257-column logits matrix would not otherwise), which is what TMA tensor maps
    and the vectorised row kernels need. The padding columns are not initialised."""
    pitch = pitch or (cols + 63) // 64 * 64
    return torch.empty(rows, pitch, device=device, dtype=dtype)[:, :cols]


class _XentFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, logits, targets, ignore_index, inplace_grad):
        V = logits.shape[-1]
        l2 = logits.reshape(-1, V)
        if l2.stride(-1) != 1 or l2.stride(0) % 8 or l2.stride(0) < (V + 7) // 8 * 8 or l2.data_ptr() % 16:
            # rows must start on 16-byte boundaries and leave room for the last vector: copy into a padded buffer
            l2 = _padded_rows(l2.shape[0], V, l2.device, l2.dtype).copy_(l2)
        T = l2.shape[0]
        tg = targets.reshape(-1).to(torch.int64).contiguous()
        n_valid = None
        if ignore_index is not None:
            n_valid = (tg != ignore_index).sum().clamp(min=1).to(torch.float32)
        loss_rows = torch.empty(T, dtype=torch.float32, device=logits.device)
        need_grad = logits.requires_grad
        dl = None
        if need_grad:
            dl = l2 if inplace_grad else _padded_rows(T, V, l2.device, l2.dtype, pitch=l2.stride(0))
        # the 1/N of the mean is folded in here; backward only multiplies by the incoming scalar
        scale = 1.0 / T if n_valid is None else None
        if scale is None:
            scale = 1.0 / float(n_valid.item())
        _rc(_lib.cuda_lib().gf_xent_fused(l2.data_ptr(), tg.data_ptr(), loss_rows.data_ptr(),
                                          dl.data_ptr() if dl is not None else None, T, V, l2.stride(0), scale,
                                          ignore_index if ignore_index is not None else -(1 << 62),
                                          _lib.status_word(l2.device).data_ptr(), _lib.stream_ptr()), "gf_xent_fused")
        loss = loss_rows.sum() * scale
        ctx.save_for_backward(dl if dl is not None else torch.empty(0, device=logits.device))
        ctx.shape = logits.shape
        return loss

    @staticmethod
    def backward(ctx, dloss):
        (dl,) = ctx.saved_tensors
        if dl.numel() == 0:
            return None, None, None, None
        g = dl.view(ctx.shape)
        # dloss is 1.0 for a plain loss.backward(): scale only when it is something else. On the GPU the kernel
        # reads the scalar and returns at once when it is 1, so the host never waits for the value (a host read
        # here would stall every backward pass and cannot be recorded in a CUDA graph).
        if dloss.numel() != 1:
            return g * dloss.to(g.dtype), None, None, None
        g2 = g.reshape(-1, g.shape[-1])
        if g.is_cuda and g.dtype == torch.bfloat16 and g2.stride(1) == 1 and g2.data_ptr() == g.data_ptr() \
                and g.data_ptr() % 16 == 0:
            # rows may have a padded pitch: the span from the first to the last element is scaled, padding included
            span = (g2.shape[0] - 1) * g2.stride(0) + g2.shape[1]
            _lib.check_rc(_lib.cuda_lib().gf_scale_by_dev_scalar(g.data_ptr(), span,
                                                                 dloss.float().data_ptr(), _lib.stream_ptr()),
                          "gf_scale_by_dev_scalar")
            return g, None, None, None
        return (g * dloss.to(g.dtype) if float(dloss) != 1.0 else g), None, None, None


def cross_entropy(logits, targets, ignore_index: int | None = None, inplace_grad: bool = False):
    """Mean softmax cross-entropy over rows. On CUDA bf16 the forward also produces the logits
    gradient in the same pass (``inplace_grad=True`` overwrites ``logits`` with it).
    ``ignore_index=None`` promises that every target is a class id, which avoids a host sync."""
    V = logits.shape[-1]
    if _cuda_bf16(logits) and (V + 7) // 8 * 16 <= 200 * 1024:
        return _XentFn.apply(logits, targets, ignore_index, inplace_grad)
    return F.cross_entropy(logits.reshape(-1, V).float(), targets.reshape(-1).long(),
                           ignore_index=-100 if ignore_index is None else ignore_index)


# ------------------------------------------------------------------------------------------ attention
def attention_ref(q, k, v, causal=True, scale=None):
    """fp32 reference SDPA. q: [B,S,Hq,D]; k, v: [B,S,Hkv,D]."""
    B, S, Hq, D = q.shape
    Hkv = k.shape[2]
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    qf = q.float().transpose(1, 2)
    kf = k.float().transpose(1, 2).repeat_interleave(Hq // Hkv, dim=1)
    vf = v.float().transpose(1, 2).repeat_interleave(Hq // Hkv, dim=1)
    s = torch.matmul(qf, kf.transpose(-1, -2)) * scale
    if causal:
        mask = torch.ones(S, k.shape[1], dtype=torch.bool, device=q.device).tril()
        s = s.masked_fill(~mask, float("-inf"))
    p = torch.softmax(s, dim=-1)
    return torch.matmul(p, vf).transpose(1, 2).to(q.dtype)


def _rows_view(t):
    """[B,S,H,D] -> (2-D alias [B*S, H*D] pitch) requirements: unit stride over D, heads packed."""
    B, S, H, D = t.shape
    if t.stride(3) != 1 or t.stride(2) != D or t.stride(0) != S * t.stride(1):
        return None
    return t.stride(1)


class _FlashAttnFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, q, k, v, causal, scale):
        B, S, Hq, D = q.shape
        Hkv = k.shape[2]
        ldq, ldk, ldv = _rows_view(q), _rows_view(k), _rows_view(v)
        if ldq is None or (ldq % 8):
            q = q.contiguous(); ldq = Hq * D
        if ldk is None or (ldk % 8):
            k = k.contiguous(); ldk = Hkv * D
        if ldv is None or (ldv % 8):
            v = v.contiguous(); ldv = Hkv * D
        o = torch.empty((B, S, Hq, D), dtype=q.dtype, device=q.device)
        lse = torch.empty((B, Hq, S), dtype=torch.float32, device=q.device)
        lib = _lib.cuda_lib()
        _rc(_lib.flash_fwd_fn()(q.data_ptr(), k.data_ptr(), v.data_ptr(), o.data_ptr(), lse.data_ptr(), B, S, Hq,
                                  Hkv, D, ldq, ldk, ldv, Hq * D, float(scale), 1 if causal else 0,
                                  _lib.status_word(q.device).data_ptr(), _lib.stream_ptr()), "gf_flash_attn_fwd")
        ctx.save_for_backward(q, k, v, o, lse)
        ctx.args = (causal, scale, ldq, ldk, ldv)
        return o

    @staticmethod
    def backward(ctx, do):
        q, k, v, o, lse = ctx.saved_tensors
        causal, scale, ldq, ldk, ldv = ctx.args
        B, S, Hq, D = q.shape
        Hkv = k.shape[2]
        if S % 128:
            raise RuntimeError("flash attention backward needs a sequence length that is a multiple of 128")
        do = do.contiguous()
        # one packed gradient buffer [B,S,(Hq+2Hkv),D] so a fused QKV projection sees a single tensor
        dqkv = torch.empty((B, S, Hq + 2 * Hkv, D), dtype=q.dtype, device=q.device)
        dq, dk, dv = dqkv[:, :, :Hq], dqkv[:, :, Hq:Hq + Hkv], dqkv[:, :, Hq + Hkv:]
        ldg = (Hq + 2 * Hkv) * D
        _lib.flash_attn_backward(q, k, v, o, do, lse, dq, dk, dv, B, S, Hq, Hkv, D,
                                 dict(q=ldq, k=ldk, v=ldv, o=Hq * D, do=Hq * D, dq=ldg, dk=ldg, dv=ldg), scale, causal)
        return dq, dk, dv, None, None


class _SplitQKVFn(torch.autograd.Function):
    """``qkv [B, S, H + 2 Hk, D] -> q, k, v`` as views. Plain slicing gives the same forward, but its backward pads
    each of the three gradients to the full shape with zeros and adds them (six passes over the packed tensor); the
    attention backward already writes its three gradients into one packed buffer, which this function recognises
    and hands on as it is."""

    @staticmethod
    def forward(ctx, qkv, H, Hk):
        ctx.H, ctx.Hk = H, Hk
        return qkv[:, :, :H], qkv[:, :, H:H + Hk], qkv[:, :, H + Hk:]

    @staticmethod
    def backward(ctx, dq, dk, dv):
        H, Hk = ctx.H, ctx.Hk
        if dq is None or dk is None or dv is None:
            ref = next(t for t in (dq, dk, dv) if t is not None)
            B, S, _, D = ref.shape
            dq = dq if dq is not None else ref.new_zeros(B, S, H, D)
            dk = dk if dk is not None else ref.new_zeros(B, S, Hk, D)
            dv = dv if dv is not None else ref.new_zeros(B, S, Hk, D)
        B, S, _, D = dq.shape
        G = H + 2 * Hk
        packed = (S * G * D, G * D, D, 1)
        same = (dq.untyped_storage().data_ptr() == dk.untyped_storage().data_ptr() == dv.untyped_storage().data_ptr()
                and dq.stride() == packed and dk.stride() == packed and dv.stride() == packed
                and dk.storage_offset() == dq.storage_offset() + H * D
                and dv.storage_offset() == dq.storage_offset() + (H + Hk) * D)
        if same:
            return dq.as_strided((B, S, G, D), packed, dq.storage_offset()), None, None
        return torch.cat((dq, dk, dv), 2), None, None


def split_qkv(qkv: torch.Tensor, num_heads: int, num_kv_heads: int):
    """Views ``q [B,S,H,D]``, ``k``, ``v [B,S,Hk,D]`` of a packed projection output ``[B,S,H+2Hk,D]``."""
    if torch.is_grad_enabled() and qkv.requires_grad:
        return _SplitQKVFn.apply(qkv, num_heads, num_kv_heads)
    H, Hk = num_heads, num_kv_heads
    return qkv[:, :, :H], qkv[:, :, H:H + Hk], qkv[:, :, H + Hk:]


def flash_attention(q, k, v, causal: bool = True, scale: float | None = None):
    """Attention over ``q [B,S,Hq,D]``, ``k/v [B,S,Hkv,D]`` (views into a packed QKV tensor are fine).
    head_dim 64 or 128 on the tcgen05 kernels; anything else uses the fp32 reference math."""
    D = q.shape[-1]
    scale = scale if scale is not None else 1.0 / math.sqrt(D)
    if _cuda_bf16(q, k, v) and D in (64, 128) and q.shape[1] == k.shape[1]:
        return _call(_FlashAttnFn, q, k, v, causal, scale)
    return attention_ref(q, k, v, causal, scale)


# ------------------------------------------------------------------------------------------ a whole pre-norm block
@functools.lru_cache(maxsize=1024)
def _block_bytes(device: int, sizes) -> tuple:
    """Bytes of the block's buffers on a device (the number of SMs decides which products split K): what a forward pass leaves for
    the backward pass, the latter's workspace, the former's, and the one of a forward pass that leaves nothing. -1: sizes
    that are not taken."""
    return tuple(_lib.cuda_lib().gf_gpt_block_bytes(which, *sizes) for which in range(4))


@functools.lru_cache(maxsize=1024)
def _block_parts(B, S, E, F, H, Hk):
    """The tensors in the buffer that a forward pass leaves for its backward pass: first byte, last, type and shape of each."""
    first = (ctypes.c_longlong * 10)()
    _rc(_lib.cuda_lib().gf_gpt_block_parts(first, B, S, E, F, H, Hk), "gf_gpt_block_parts")
    bf16, fp32 = torch.bfloat16, torch.float32
    kinds = ((bf16, (B, S, E)), (fp32, (2, B * S)), (bf16, (B, S, H + 2 * Hk, E // H)), (bf16, (B, S, E)), (fp32, (B, H, S)),
             (bf16, (B, S, E)), (bf16, (B, S, E)), (fp32, (2, B * S)), (bf16, (B, S, F)), (bf16, (B, S, F)))
    return [(n, n + math.prod(s) * t.itemsize, t, s) for n, (t, s) in zip(first, kinds)]


# private name of torch: the hooks that saved tensors go through, if any; without the name they count as present
_SAVED_HOOKS = getattr(torch._C._autograd, "_top_saved_tensors_default_hooks", None)


def _saved_tensors_are_hooked() -> bool:
    return _SAVED_HOOKS is None or _SAVED_HOOKS(True) is not None


def _dense16(t):
    """``t`` itself where it is dense on a 16-byte boundary, else a copy that is."""
    t = _dense(t)
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _pointers(ts):
    return (ctypes.c_void_p * len(ts))(*[None if t is None else t.data_ptr() for t in ts])


class _GPTBlockFn(torch.autograd.Function):
    """See :func:`gpt_block`. The launches of a pass are one call; what the backward pass reads again is one buffer, which hooks on
    saved tensors get as the typed tensors that it holds: a hook may do with a tensor what its type and shape tell it."""

    @staticmethod
    def forward(ctx, x, sizes, eps1, eps2, causal, *params):
        y, dev, graph = torch.empty_like(x), x.device, type(ctx) is not _NoGraph
        nsaved, nback, nws, alone = _block_bytes(dev.index, sizes)
        if not graph:                      # the layers' results share a small workspace
            nsaved, nws = 0, alone
        saved = torch.empty(nsaved, dtype=torch.uint8, device=dev) if nsaved else None
        ws = torch.empty(nws, dtype=torch.uint8, device=dev) if nws else None
        _rc(_lib.cuda_lib().gf_gpt_block_fwd(x.data_ptr(), _pointers(params), y.data_ptr(), None if saved is None else saved.data_ptr(),
                                             nsaved, None if ws is None else ws.data_ptr(), nws, *sizes, causal, eps1, eps2,
                                             _lib.status_word(dev).data_ptr(), _lib.stream_ptr()), "gf_gpt_block_fwd")
        hooked = graph and _saved_tensors_are_hooked()
        if hooked:
            ctx.save_for_backward(x, *(saved[n:e].view(t).view(s) for n, e, t, s in _block_parts(*sizes)), *params)
        else:
            ctx.save_for_backward(x, saved, *params)
        ctx.args = sizes, causal, hooked, nback
        return y

    @staticmethod
    def backward(ctx, dy):
        sizes, causal, hooked, nws = ctx.args
        parts = None
        if not hooked:
            x, saved, *params = ctx.saved_tensors
            at, nsaved = saved.data_ptr(), saved.numel()
        else:
            x, *kept = ctx.saved_tensors
            kinds, at, nsaved = _block_parts(*sizes), None, 0
            kept, params = kept[:len(kinds)], kept[len(kinds):]
            for k, (_, _, t, s) in zip(kept, kinds):
                if k.dtype is not t or k.shape != s or k.device != x.device:
                    raise RuntimeError(f"a hook returned a saved tensor of {k.dtype} {list(k.shape)} on {k.device} for one of {t} "
                                       f"{list(s)} on {x.device}")
            # hooks may bring all of them back in another layout
            kept, x, params = [_dense16(k) for k in kept], _dense16(x), [None if p is None else _dense16(p) for p in params]
            parts = _pointers(kept)
        dy = _dense16(dy)
        dx = torch.empty_like(x)
        # the norms' kernels always write theirs
        grads = [torch.empty_like(p) if p is not None and (need or i in (0, 6)) else None
                 for i, (p, need) in enumerate(zip(params, ctx.needs_input_grad[5:]))]
        ws = torch.empty(nws, dtype=torch.uint8, device=x.device)
        _rc(_lib.cuda_lib().gf_gpt_block_bwd(x.data_ptr(), _pointers(params), dy.data_ptr(), at, nsaved, parts, dx.data_ptr(),
                                             _pointers(grads), ws.data_ptr(), nws, *sizes, causal,
                                             _lib.status_word(x.device).data_ptr(), _lib.stream_ptr()), "gf_gpt_block_bwd")
        return (dx, None, None, None, None, *grads)


def gpt_block(x, params, sizes, eps1: float, eps2: float, causal: bool):
    """``h = x + Wo attention(LN1(x) Wqkv^T + bqkv) + bo``, ``y = h + W2 gelu(LN2(h) W1^T + b1) + b2`` on the kernels of the layers,
    all launches of a pass from one call of the kernel library. ``params``: ln1 weight and bias, Wqkv, bqkv, Wo, bo, ln2
    weight and bias, W1, b1, W2, b2 (biases may be ``None``); ``sizes``: batch, sequence, width, inner width, heads, KV heads."""
    y = _call(_GPTBlockFn, x, sizes, float(eps1), float(eps2), 1 if causal else 0, *params)
    if _lib.DEBUG_SYNC:
        _lib.check_status()
    return y


def gpt_block_ok(x, params, sizes) -> bool:
    """Whether :func:`gpt_block` takes these operands: dense bf16 CUDA tensors of the sizes, on 16-byte boundaries, with head
    sizes and (where there is a gradient) a sequence that the attention kernels have, and nothing that follows the layers'
    own calls."""
    B, S, E, F_, H, Hk = sizes
    if _observed():                         # before anything asks a tensor for its memory: transformed ones have none
        return False
    if type(x) is not torch.Tensor or not _cuda_bf16(x) or not x.is_contiguous() or x.data_ptr() % 16 or E > 8192 or F_ > 8192 \
            or (H + 2 * Hk) * (E // H) > 8192 or _block_bytes(x.device.index, sizes)[0] < 0 or x.device.index != torch.cuda.current_device():
        return False
    P = (H + 2 * Hk) * (E // H)
    shapes = ((E,), (E,), (P, E), (P,), (E, E), (E,), (E,), (E,), (F_, E), (F_,), (E, F_), (E,))
    grad = False
    for p, s in zip(params, shapes):
        if p is None:
            if len(s) == 2:
                return False
        elif type(p) not in (torch.Tensor, torch.nn.Parameter) or p.shape != s or p.dtype is not torch.bfloat16 \
                or p.device != x.device or not p.is_contiguous() or p.data_ptr() % 16:
            return False
        else:
            grad = grad or p.requires_grad
    if (grad or x.requires_grad) and torch.is_grad_enabled() and S % 128:
        return False                        # the layers say what they miss
    return os.environ.get("GF_FA_FWD", "3") == "3" and os.environ.get("GF_FA_BWD", "3") != "1"
