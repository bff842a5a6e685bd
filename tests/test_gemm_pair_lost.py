"""Products that a cut on pairs of blocks makes slower are left as they are (csrc/bindings.cpp: pair_choice)."""
import pytest

from nanorlhf_b200 import _C

SMS, FITS = 148, [0, 0, 74, 45, 33, 26, 22, 15, 15]         # a B200: clusters of 2 .. 8 blocks that run at a time


@pytest.mark.parametrize("M,N,K", [
    (39, 3584, 1536), (128, 3584, 1536), (1, 4096, 1792), (128, 18944, 18944),                   # half of a pair without work
    (493, 1536, 1536), (541, 1536, 2048), (1131, 1024, 3072), (154, 3072, 1408),                 # contractions too short to pay for the sum
    (1000, 3584, 151936), (5000, 1536, 151936), (1500, 3584, 151936), (256, 896, 34816),                   # a sum, or rounds, that cost more
])
def test_not_cut_on_pairs(M, N, K):
    assert _C.gemm_tc_pair_choice(M, N, K, SMS, FITS)[1] == 1


def test_what_passes_through_a_workspace_runs_at_once():
    taken = 0
    for M in range(129, 6000, 173):
        for N in (128, 512, 896, 1024, 1536, 2048, 3584, 4096):
            for K in (34816, 65536, 151936):
                bn, n, clusters = _C.gemm_tc_pair_choice(M, N, K, SMS, FITS)
                if n > 1 and not clusters:
                    taken += 1
                    assert n * -(-M // 256) * -(-N // bn) <= SMS // 2
    assert taken > 50
