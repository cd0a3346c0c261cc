"""Which products split K over CTAs: the rule of the kernel library, asked by the host code that allocates the workspace."""
import pytest

from ghost_flow_b200.ops.gemm import _splits

K_MAJOR = dict(a_mn_major=False, b_mn_major=False, aligned=True, accumulate=False, relu=False)


def splits(M, N, K, **kw):
    return _splits(M, N, K, **{**K_MAJOR, **kw})


# measured on both paths; the few-row kernel where it was at least as fast
@pytest.mark.parametrize("M,N,K,want", [
    (1, 4096, 4096, False), (8, 4096, 11008, False), (8, 4096, 16384, False), (8, 2048, 8192, False), (8, 64, 6144, False),
    (8, 1024, 8192, True), (8, 512, 16384, True), (1, 2048, 11008, True), (1, 16, 65536, True), (8, 4096, 32768, True),
    (9, 64, 4096, False), (16, 4096, 8192, False), (16, 8192, 14336, False), (16, 2048, 8192, True), (16, 4096, 11008, True),
    (9, 128, 65536, True), (17, 4096, 4096, True), (17, 4096, 2040, False), (64, 28672, 8192, False), (64, 8192, 14336, True)])
def test_split_where_it_is_faster(M, N, K, want):
    assert splits(M, N, K) == want


def test_forms_that_never_or_always_split():
    for kw in (dict(accumulate=True), dict(relu=True)):
        assert not splits(8, 512, 16384, **kw) and not splits(64, 512, 16384, **kw)
    # operands that the few-row kernel does not read
    for kw in (dict(a_mn_major=True), dict(b_mn_major=True), dict(aligned=False)):
        assert splits(8, 4096, 4096, **kw)
    assert splits(8, 4096, 4100)
