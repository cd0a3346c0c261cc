"""Sizes of the buffers of the one-call GPT block: asked of the kernel library, which refuses smaller ones before it launches."""
import ctypes
import os
import subprocess
import sys

import pytest

from ghost_flow_b200.ops import _lib

SIZES = 8, 1024, 768, 3072, 12, 12          # products with sums of parts of K as workspace, in both directions
BAD_ARG = -1


def _bytes(which):
    return _lib.cuda_lib().gf_gpt_block_bytes(which, *SIZES)


def _call(saved_bytes, ws_bytes, backward=False, saved=1 << 20):
    """No pointer is looked at before the sizes are."""
    lib, p = _lib.cuda_lib(), 1 << 20
    table = (ctypes.c_void_p * 12)(*[p] * 12)
    if backward:
        return lib.gf_gpt_block_bwd(p, table, p, saved, saved_bytes, None, p, table, p, ws_bytes, *SIZES, 1, None, None)
    return lib.gf_gpt_block_fwd(p, table, p, saved, saved_bytes, p, ws_bytes, *SIZES, 1, 1e-5, 1e-5, None, None)


@pytest.mark.parametrize("short", [(1, 0), (0, 1), (1, 1)])
def test_buffers_that_are_too_small_are_refused(short):
    assert _call(_bytes(0) - 256 * short[0], _bytes(2) - short[1]) == BAD_ARG
    assert _call(_bytes(0) - 256 * short[0], _bytes(1) - short[1], backward=True) == BAD_ARG
    if short[1]:
        assert _call(0, _bytes(3) - 1, saved=None) == BAD_ARG


def test_parts_of_the_buffer_are_apart_and_inside_it():
    from ghost_flow_b200.ops.fused import _block_parts

    for sizes in (SIZES, (1, 128, 128, 136, 2, 2), (3, 100, 256, 512, 4, 2)):
        end = 0
        for first, last, _, _ in _block_parts(*sizes):
            assert first % 256 == 0 and end <= first < last
            end = last
        assert end <= _lib.cuda_lib().gf_gpt_block_bytes(0, *sizes) < end + 256


def test_without_a_gradient_less_is_held():
    """The layers' results share three buffers and the output then."""
    B, S, E, F, _, _ = SIZES
    assert _bytes(3) <= _bytes(2) + 2 * B * S * (E + 2 * F) + 1024 < _bytes(0) / 1.6


def test_the_environment_is_read_once():
    """A workspace that was sized before a variable changes is the one that the call takes after it."""
    code = """
import ctypes, os
from ghost_flow_b200.ops import _lib
lib, libc = _lib.cuda_lib(), ctypes.CDLL(None)
ask = lambda: [lib.gf_gpt_block_bytes(w, 8, 1024, 768, 3072, 12, 12) for w in range(4)]
before = ask()
libc.setenv(b"GF_GEMM_2SM", b"0", 1)
assert ask() == before, (before, ask())
libc.unsetenv(b"GF_GEMM_2SM")
assert ask() == before
"""
    for env in ({}, {"GF_GEMM_2SM": "0"}):
        env = {**{k: v for k, v in os.environ.items() if k != "GF_GEMM_2SM"}, **env}
        subprocess.run([sys.executable, "-c", code], check=True, env=env, cwd=os.path.dirname(os.path.dirname(__file__)))
