"""Which steps of the delta-rule scan go four tokens at a time, and which stay with the column-resident form that serves them better."""
import pytest

from nanorlhf_b200 import _C


@pytest.mark.parametrize("E,T,D,Dv,blocked", [
    (1, 1, 128, 128, False), (256, 256, 128, 128, False),                                  # decoding
    (1, 20, 64, 64, True), (1, 19, 64, 64, False), (16, 320, 128, 128, True), (16, 319, 128, 128, False),
    (16, 16 * 2048, 128, 128, True), (65, 64 + 2000, 128, 128, True), (65, 64 + 700, 128, 128, False),
    (64, 64 * 128, 33, 33, True), (64, 64 * 128, 32, 32, False), (1, 2000, 16, 64, False), (256, 256 * 12, 8, 8, False),      # few state rows
    (1, 12, 32, 320, True), (1, 11, 32, 320, False), (16, 16 * 12, 128, 512, True),        # more columns than the column form takes
    (1, 2000, 129, 64, False),
])
def test_form_of_a_step(E, T, D, Dv, blocked):
    assert bool(_C.delta_scan_blocked(E, T, D, Dv)) == blocked
