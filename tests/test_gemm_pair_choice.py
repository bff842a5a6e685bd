"""Which products are cut into ranges of their contraction on pairs of blocks (csrc/bindings.cpp): what the rule says at the sizes where it was measured, and
that everything that it says can be launched."""
import pytest

from nanorlhf_b200 import _C

SMS, FITS = 148, [0, 0, 74, 45, 33, 26, 22, 15, 15]         # a B200: clusters of 2 .. 8 blocks that run at a time


def _choice(M, N, K):
    return _C.gemm_tc_pair_choice(M, N, K, SMS, FITS)


@pytest.mark.parametrize("M,N,K,want", [
    (1024, 1536, 8960, (192, 2, True)), (900, 1536, 8960, (192, 2, True)), (512, 1536, 8960, (256, 4, True)), (768, 1536, 8960, None), (256, 1536, 8960, None),
    (8, 1536, 8960, None), (6601, 1536, 8960, None), (1024, 1536, 1536, None), (1024, 2048, 1536, None), (256, 3584, 18944, (256, 4, True)), (100, 1536, 151936, None),
    (300, 1536, 151936, None), (768, 1536, 151936, (256, 4, False)), (1000, 1536, 151936, (256, 3, False)), (6001, 1536, 151936, None), (4096, 64, 8960, None),
])
def test_choice(M, N, K, want):
    bn, n, clusters = _choice(M, N, K)
    assert (None if n == 1 else (bn, n, clusters)) == want


def test_every_choice_can_be_launched_as_it_is():
    taken = 0
    for M in (1, 8, 100, 128, 300, 512, 700, 1000, 2000, 3000, 6000, 9400):
        for N in (8, 64, 72, 256, 1024, 1536, 3584, 8960):
            for K in [*range(64, 9000, 192), 18944, 32768, 65536, 151936]:
                (bn, n, clusters), blocks = _choice(M, N, K), -(-K // 64)
                if n == 1:
                    continue
                taken += 1
                tiles = -(-M // 256) * -(-N // bn)
                assert bn in (128, 192, 256) and N > 64
                assert -(-blocks // -(-blocks // n)) == n and blocks >= 4 * n            # no range is empty
                if clusters:
                    assert 2 * n <= 8 and tiles <= FITS[2 * n]
                else:
                    assert n * tiles * 256 * bn * 4 <= 128 << 20                         # workspace of a call
    assert taken > 100
