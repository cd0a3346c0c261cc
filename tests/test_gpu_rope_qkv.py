"""Rotary embedding of a packed projection in one launch (``rope_qkv``) against split + ``rope`` one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _close(a, b):
    # the same fp32 formula, contracted differently at most: equal up to one bf16 rounding (2^-8 relative, and 2^-8 of a
    # product that cancelled)
    return torch.allclose(a.float(), b.float(), rtol=2 ** -7, atol=2 ** -7)


@pytest.mark.parametrize("B,S,H,Hk,D", [(1, 1, 1, 1, 16), (2, 37, 3, 3, 48), (2, 5, 8, 2, 64), (1, 130, 40, 8, 128), (3, 1, 4, 4, 256)])
@pytest.mark.parametrize("interleaved", [False, True])
def test_rope_qkv_forward_and_backward(B, S, H, Hk, D, interleaved):
    from ghost_flow_b200 import ops

    pos = 3
    cos, sin = ops.rope_tables(S + pos, D, 1e4, "cuda")
    x = torch.randn(B, S, H + 2 * Hk, D, device="cuda", dtype=torch.bfloat16)
    a, b = x.clone().requires_grad_(), x.clone().requires_grad_()
    got = ops.rope_qkv(a, H, Hk, cos, sin, interleaved, pos)
    q, k, v = ops.split_qkv(b, H, Hk)
    want = ops.rope(q, cos, sin, interleaved, pos), ops.rope(k, cos, sin, interleaved, pos), v
    # gradients as three tensors, one of them strided so that it has to be copied first
    gs = [torch.randn_like(t) for t in want]
    gs[1] = torch.randn(B, Hk, S, D, device="cuda", dtype=torch.bfloat16).transpose(1, 2)
    for g, w in zip(got, want):
        assert _close(g, w)
    torch.autograd.backward(got, gs)
    torch.autograd.backward(want, gs)
    assert _close(a.grad, b.grad)
    with torch.no_grad():
        for g, w in zip(ops.rope_qkv(x, H, Hk, cos, sin, interleaved, pos), want):
            assert _close(g, w)


@pytest.mark.parametrize("B,S,H,Hk,D", [(3, 1, 4, 2, 64), (2, 7, 8, 8, 128), (1, 1, 5, 5, 24)])
@pytest.mark.parametrize("layout", ["plain", "heads_first"])
def test_rope_qkv_to_cache(B, S, H, Hk, D, layout):
    from ghost_flow_b200 import ops

    pos, n = 11, 32
    cos, sin = ops.rope_tables(n, D, 1e4, "cuda")
    qkv = torch.randn(B, S, H + 2 * Hk, D, device="cuda", dtype=torch.bfloat16)
    if layout == "plain":
        caches = [torch.randn(B, n, Hk, D, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
    else:                                  # a layout the kernel does not write: takes the assignments
        caches = [torch.randn(B, Hk, n, D, device="cuda", dtype=torch.bfloat16).transpose(1, 2) for _ in range(2)]
    want = [c.clone() for c in caches]
    with torch.no_grad():
        q = ops.rope_qkv_to_cache(qkv, H, Hk, cos, sin, *caches, False, pos)
        qs, ks, vs = ops.split_qkv(qkv, H, Hk)
        want[0][:, pos:pos + S] = ops.rope(ks, cos, sin, False, pos)
        want[1][:, pos:pos + S] = vs
    assert _close(q, ops.rope(qs, cos, sin, False, pos))
    for c, w in zip(caches, want):
        assert _close(c, w)
        rest = torch.ones(n, dtype=torch.bool)
        rest[pos:pos + S] = False
        assert torch.equal(c[:, rest], w[:, rest])


def test_positions_outside_the_tables_are_refused_before_any_launch():
    from ghost_flow_b200 import ops
    from ghost_flow_b200.ops import _lib, raw

    qkv = torch.randn(1, 4, 6, 64, device="cuda", dtype=torch.bfloat16)
    kc, vc = (torch.zeros(1, 32, 2, 64, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    tables = [(*ops.rope_tables(8, 64, 1e4, "cuda"), 5), (*ops.rope_tables(8, 64, 1e4, "cuda"), -1),
              (*ops.rope_tables(8, 128, 1e4, "cuda"), 0), (*ops.rope_tables(8, 64, 1e4, "cpu"), 0)]
    n0 = _lib.launch_count()
    for cos, sin, pos in tables:
        with torch.no_grad(), pytest.raises(ValueError):
            ops.rope_qkv_to_cache(qkv, 2, 2, cos, sin, kc, vc, False, pos)
        with pytest.raises(ValueError):
            ops.rope_qkv(qkv, 2, 2, cos, sin, False, pos)
        with pytest.raises(ValueError):
            ops.rope(qkv, cos, sin, False, pos)
        with pytest.raises(ValueError):
            raw.rope_(qkv.view(4, 6, 64), cos, sin, 4, False, pos)
    assert _lib.launch_count() == n0 and not kc.any() and not vc.any()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float64])
def test_tables_of_another_type_give_the_same_rotation(dtype):
    from ghost_flow_b200 import ops

    x = torch.randn(2, 5, 6, 64, device="cuda", dtype=torch.bfloat16)
    cos, sin = (t.to(dtype) for t in ops.rope_tables(8, 64, 1e4, "cuda"))
    got, want = ops.rope_qkv(x, 2, 2, cos, sin, False, 3), ops.rope_qkv(x, 2, 2, cos.float(), sin.float(), False, 3)
    for g, w in zip(got, want):
        assert _close(g, w)


def test_cache_writes_are_visible_to_autograd_and_to_dispatch_modes():
    from torch.utils._python_dispatch import TorchDispatchMode

    from ghost_flow_b200 import ops

    cos, sin = ops.rope_tables(8, 64, 1e4, "cuda")
    qkv = torch.randn(1, 1, 6, 64, device="cuda", dtype=torch.bfloat16)
    kc, vc = (torch.randn(1, 8, 2, 64, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    w = torch.ones_like(kc, requires_grad=True)
    for saved in (kc, vc):
        y = (saved * w).sum()
        with torch.no_grad():
            ops.rope_qkv_to_cache(qkv, 2, 2, cos, sin, kc, vc, False, 3)
        with pytest.raises(RuntimeError, match="modified by an inplace operation"):
            y.backward()
    with torch.inference_mode():
        ic = torch.zeros_like(kc), torch.zeros_like(vc)
        ops.rope_qkv_to_cache(qkv, 2, 2, cos, sin, *ic, False, 3)
    assert torch.equal(ic[0][:, 3], kc[:, 3]) and torch.equal(ic[1][:, 3], vc[:, 3])

    written = []

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            if func._schema.name == "aten::copy_":
                written.append(args[0].untyped_storage().data_ptr())
            return func(*args, **(kwargs or {}))

    want = kc.clone(), vc.clone()
    with torch.no_grad(), Mode():
        ops.rope_qkv_to_cache(qkv, 2, 2, cos, sin, kc, vc, False, 3)
    assert {kc.untyped_storage().data_ptr(), vc.untyped_storage().data_ptr()} <= set(written)
    assert _close(kc, want[0]) and _close(vc, want[1])


def test_caches_whose_rows_share_memory_take_the_assignments():
    from ghost_flow_b200 import ops

    cos, sin = ops.rope_tables(8, 64, 1e4, "cuda")
    qkv = torch.randn(2, 1, 6, 64, device="cuda", dtype=torch.bfloat16)
    mk = lambda b: torch.zeros(b, 8, 2, 64, device="cuda", dtype=torch.bfloat16)  # noqa: E731
    with torch.no_grad():
        with pytest.raises(RuntimeError):                   # refused, as a write to an expanded tensor is
            ops.rope_qkv_to_cache(qkv, 2, 2, cos, sin, mk(1).expand(2, -1, -1, -1), mk(2), False, 3)
        both = mk(2)
        ops.rope_qkv_to_cache(qkv, 2, 2, cos, sin, both, both, False, 3)
    assert torch.equal(both[:, 3], qkv[:, 0, 4:])           # v is written last
