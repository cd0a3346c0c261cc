"""Layouts of a KV cache that one kernel may write in any order: no two rows share memory."""
import itertools

import pytest
import torch

from ghost_flow_b200.ops.fused import _cache_rows_apart

B, N, H, D = 3, 5, 2, 8


def _views():
    z = torch.zeros
    flat = z(4 * B * N * H * D + 64)
    yield "two tensors", (z(B, N, H, D), z(B, N, H, D))
    yield "stacked", tuple(z(2, B, N, H, D))
    yield "interleaved rows", (lambda t: (t[:, :, 0], t[:, :, 1]))(z(B, N, 2, H, D))
    yield "interleaved sequences", (lambda t: (t[:, 0], t[:, 1]))(z(B, 2, N, H, D))
    yield "tokens first", tuple(z(N, B, H, D).transpose(0, 1) for _ in range(2))
    yield "tokens first, interleaved", (lambda t: (t[:, :, 0].transpose(0, 1), t[:, :, 1].transpose(0, 1)))(z(N, B, 2, H, D))
    yield "part of longer caches", (z(B, 9, H, D)[:, 2:2 + N], z(7, N, H, D)[1:1 + B])
    yield "one sequence", (z(1, N, H, D), z(1, N, H, D))
    yield "one row", (z(B, 1, H, D), z(B, 1, H, D))
    yield "expanded over sequences", (z(1, N, H, D).expand(B, N, H, D), z(B, N, H, D))
    yield "expanded over tokens", (z(B, N, H, D), z(B, 1, H, D).expand(B, N, H, D))
    yield "the same twice", (lambda t: (t, t))(z(B, N, H, D))
    for off in (1, H * D - 1, H * D, H * D + 8, B * N * H * D - 1, B * N * H * D):
        yield f"offset {off}", tuple(flat[o:o + B * N * H * D].view(B, N, H, D) for o in (0, off))
    for sb, sn in itertools.product((0, 8, H * D, N * H * D), repeat=2):
        yield f"strides {sb} {sn}", (flat.as_strided((B, N, H, D), (sb, sn, D, 1)), z(B, N, H, D))


def _rows(t):
    return [set(range(int(o), int(o) + H * D)) for b in range(t.shape[0]) for n in range(t.shape[1])
            for o in [t.data_ptr() // 4 + b * t.stride(0) + n * t.stride(1)]]


@pytest.mark.parametrize("name,pair", list(_views()), ids=lambda x: x if isinstance(x, str) else "")
def test_rows_apart_is_never_claimed_wrongly(name, pair):
    rows = _rows(pair[0]) + _rows(pair[1])
    apart = sum(map(len, rows)) == len(set().union(*rows))
    # every layout above that is free of overlap is also one the kernel may write
    assert _cache_rows_apart(*pair) == apart
    assert _cache_rows_apart(*pair[::-1]) == apart
