"""Which steps of the delta-rule scan with one decay per head go 32 tokens at a time."""
import pytest

from nanorlhf_b200 import _C


@pytest.mark.parametrize("E,T,heads,D,Dv,chunked", [
    (256, 256, 16, 128, 128, False), (1, 19, 1, 128, 128, False), (1, 20, 1, 33, 4, True), (1, 2000, 1, 32, 32, False), (1, 2000, 1, 132, 64, False),
    (16, 320, 16, 128, 128, True), (16, 319, 16, 128, 128, False), (65, 64 + 2000, 16, 128, 128, True),
    (9, 9 * 20, 16, 64, 64, True), (10, 10 * 20, 16, 64, 64, False), (10, 10 * 128, 16, 64, 64, True),      # 148 blocks at once, then several rounds
    (10, 10 * 47, 16, 128, 64, False), (10, 10 * 48, 16, 128, 64, True), (10, 10 * 31, 16, 64, 128, False), (10, 10 * 32, 16, 64, 128, True),
    (5, 5 * 20, 16, 64, 256, False), (4, 4 * 20, 16, 64, 256, True),                                        # two blocks of columns
])
def test_form_of_a_step(E, T, heads, D, Dv, chunked):
    assert bool(_C.delta_scan_chunked(E, T, heads, D, Dv, 148)) == chunked
