"""Into how many ranges a GEMM's contraction is cut (csrc/bindings.cpp): the number that is judged is the number that is launched."""
import pytest

from nanorlhf_b200 import _C

SMS, FITS = 148, [0, 0, 74, 45, 33, 26, 22, 15, 15]         # a B200: clusters of 2 .. 8 blocks that run at a time


def _choice(M, N, K):
    return _C.gemm_tc_split_choice(M, N, K, SMS, FITS)


def _tiles(M, N):
    return -(-M // 128) * -(-N // (64 if N <= 64 else 128))


@pytest.mark.parametrize("M,N,K,ranges", [
    (128, 1536, 1024, 1), (128, 1536, 1536, 4), (128, 1536, 2112, 4), (128, 1536, 2624, 4), (128, 1536, 3136, 7), (128, 1536, 8960, 8),
    (1024, 256, 8960, 6), (1664, 64, 1024, 4), (1664, 64, 2112, 4), (1664, 64, 3136, 7), (1664, 64, 8960, 8),
    (3300, 64, 1536, 4), (3300, 192, 1536, 1), (3300, 192, 2112, 2), (6601, 64, 1536, 2), (4700, 64, 4096, 3), (4700, 64, 8960, 4),
    (512, 1536, 8960, 3), (4096, 1536, 8960, 1), (0, 64, 4096, 1), (128, 1536, 64, 1), (9600, 128, 8960, 1),
])
def test_choice(M, N, K, ranges):
    assert _choice(M, N, K) == ranges


def test_every_choice_can_be_launched_as_it_is():
    for M in (1, 128, 1000, 2000, 3000, 4000, 6000, 9400):
        for N in (8, 64, 128, 256):
            for K in range(64, 9000, 64):
                n, blocks = _choice(M, N, K), K // 64
                if n == 1:
                    continue
                assert -(-blocks // -(-blocks // n)) == n                                # no range is empty
                assert _tiles(M, N) * n <= SMS and blocks >= 4 * n
                assert n <= 4 or _tiles(M, N) <= FITS[n]                                 # beyond four ranges only where a cluster sums them


@pytest.mark.gpu
@pytest.mark.parametrize("M,N", [(128, 1536), (1664, 64), (300, 512)])
@pytest.mark.parametrize("K", [2112, 2624, 2688, 3136, 8960])
def test_the_gpus_own_choice_leaves_no_range_empty(M, N, K):
    n, blocks = _C.gemm_tc_auto_splits(M, N, K), K // 64
    assert n > 1 and -(-blocks // -(-blocks // n)) == n
    assert n <= 4 or _tiles(M, N) <= _C.gemm_tc_split_clusters(64 if N <= 64 else 128, n)
