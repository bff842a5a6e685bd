"""Which narrow products of adapters share a launch (csrc/bindings.cpp: multi_pays), at sizes where both forms were measured."""
import pytest

from nanorlhf_b200 import _C

SMS = 148


def _factors(wide, r, tokens, narrow=None):
    return _C.gemm_tc_multi_pays(wide, narrow or [r] * len(wide), [tokens] * len(wide), SMS)


@pytest.mark.parametrize("r,tokens,shared", [(64, 60, False), (64, 1000, False), (64, 4000, False), (64, 16384, False), (32, 4000, False), (16, 60, True), (16, 4000, True), (8, 4000, True)])
def test_one_projection_of_18944_columns(r, tokens, shared):
    assert _factors([3584, 18944], r, tokens) == shared


@pytest.mark.parametrize("d,f,tokens,shared", [
    (3584, 18944, 8, False), (3584, 18944, 1000, True), (3584, 18944, 16384, True), (8192, 28672, 8, False), (8192, 28672, 1000, False), (8192, 28672, 16384, True),
    (1536, 8960, 8, True), (1536, 8960, 6601, True), (4096, 14336, 60, True), (4096, 14336, 16384, True), (896, 4864, 700, True),
])
def test_gate_up_and_down(d, f, tokens, shared):
    assert _factors([f, f, d, d, f], 64, tokens, [64, 64, 64, 128, 64]) == shared


@pytest.mark.parametrize("tokens,widths,shared", [
    (6601, [8960] * 2, True), (9000, [8960] * 2, True), (12000, [8960] * 2, False), (16384, [8960] * 2, True), (6601, [1536, 256, 256], True), (12000, [1536, 256, 256], True),
    (16384, [1536, 256, 256], False), (32768, [1536, 256, 256], False), (32768, [3584, 512, 512], False),
])
def test_inputs_of_a_group(tokens, widths, shared):
    assert _C.gemm_tc_multi_pays([tokens] * len(widths), [64] * len(widths), widths, SMS) == shared


def test_empty_products_are_left_to_the_launch():
    assert _C.gemm_tc_multi_pays([0, 0], [64, 64], [1536, 256], SMS) and _C.gemm_tc_multi_pays([64], [64], [0], SMS)
