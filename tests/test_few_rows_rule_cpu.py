"""Which kernel takes a product of few rows, and the workspace that goes with it: the rules that a product follows."""
import pytest

from ghost_flow_b200.ops import _lib
from ghost_flow_b200.ops.gemm import _workspace

FORM = dict(a_mn_major=False, b_mn_major=False, aligned=True, accumulate=False)


def few_rows(M, N, K, **kw):
    return bool(_lib.cuda_lib().gf_gemm_bf16_few_rows(M, N, K, *{**FORM, **kw}.values()))


def workspace(M, N, K, relu=False, **kw):
    return _workspace(M, N, K, *{**FORM, **kw}.values(), relu)


# 148 SMs. Measured on both kernels, with cold weights; the few-row one where it was the faster
@pytest.mark.parametrize("K,takes,leaves", [
    (2048, (), (64, 512, 4096, 6144, 8192, 16384, 32000)),
    (4096, (192, 256, 1024, 2048, 4096, 11904, 12288, 13824, 14336, 15360, 16384, 23744, 24576, 28416),
     (8, 64, 128, 4864, 6144, 7168, 8192, 9216, 10240, 11776, 18432, 20480, 22016, 23552, 28672, 32000)),
    (5120, (128, 192, 4096, 12288, 15360), (8, 64, 96, 5120, 6144, 8192, 10240, 20480, 32000)),
    (8192, (8, 64, 128, 512, 4096, 5120, 12288, 24576), (6144, 8192, 10240, 20480, 22016, 28672, 32000)),
    (14336, (8, 64, 512, 4096, 5120, 12288, 16384), (6144, 7168, 8192, 10240, 20480, 22016, 32000))])
@pytest.mark.parametrize("M", [1, 8])
def test_up_to_eight_rows(M, K, takes, leaves):
    assert [few_rows(M, n, K) for n in (*takes, *leaves)] == [True] * len(takes) + [False] * len(leaves)


@pytest.mark.parametrize("K,takes,leaves", [
    (1024, (), (64, 4096, 16384)), (2048, (11008, 12288, 16384, 32000), (64, 512, 4096, 6144, 8192)),
    (3072, (6144, 8192, 12288, 24576), (64, 128)), (4096, (128, 192, 512, 4096, 6144, 12288, 32000), (8, 64, 96)),
    (5120, (8, 64, 512, 8192, 32000), ()), (11008, (8, 64, 4096, 22016), ())])
@pytest.mark.parametrize("M", [9, 16])
def test_up_to_sixteen_rows(M, K, takes, leaves):
    assert [few_rows(M, n, K) for n in (*takes, *leaves)] == [True] * len(takes) + [False] * len(leaves)


@pytest.mark.parametrize("M,N,K,want", [
    (17, 64, 64, True), (32, 32000, 8192, True), (33, 512, 504, False), (33, 512, 512, True), (64, 24576, 4096, True),
    (64, 28672, 4096, False), (65, 512, 4096, False)])
def test_more_rows(M, N, K, want):
    assert few_rows(M, N, K) == want


def test_forms_that_the_kernel_does_not_read():
    for kw in (dict(a_mn_major=True), dict(b_mn_major=True), dict(aligned=False), dict(accumulate=True)):
        assert few_rows(16, 4096, 4096) and not few_rows(16, 4096, 4096, **kw)
    assert not few_rows(16, 4096, 4100)


def test_workspaces():
    # few-row products take none; products of whole tiles with few of them and a long K take one of every part of K; others with
    # fewer tiles yet one in all
    assert workspace(16, 4096, 4096) == workspace(8, 512, 8192) == workspace(64, 4096, 8192) == workspace(8, 64, 4096) == 0
    for M, N in ((2304, 768), (3072, 768), (768, 3072), (1600, 1600)):
        parts, rest = divmod(workspace(M, N, 8192), M * N)
        assert 2 <= parts <= 4 and rest == 0
        assert workspace(M, N, 8192, accumulate=True) == workspace(M, N, 8192, relu=True) == 0
    assert workspace(768, 768, 8192) == 768 * 768 and workspace(100, 512, 8192) == 100 * 512
    assert workspace(8, 512, 16384, b_mn_major=True) == 8 * 512
    assert workspace(4096, 4096, 8192) == workspace(2304, 768, 1024) == 0
