"""How the tcgen05 paged attention cuts a step into items: full tiles where portions are long, an item for every SM where they are many and short."""
import random

import pytest

from nanorlhf_b200 import _C

SMS = 148


def _items(T, E, Hq, Hkv):
    qt = _C.window_attention_tc_tokens(T, E, Hq, Hkv, SMS)
    hb = min(128, Hq // Hkv)
    heads = Hkv * -(-(Hq // Hkv) // hb)
    return qt, 128 // hb, -(-T // (2 * qt)) * heads


@pytest.mark.parametrize("E,n,Hq,Hkv", [(64, 4, 16, 16), (64, 2, 16, 8), (200, 2, 8, 8), (64, 4, 4, 4), (64, 8, 16, 4), (64, 2, 32, 8)])
def test_many_short_portions_reach_all_sms(E, n, Hq, Hkv):
    qt, most, items = _items(E * n, E, Hq, Hkv)
    assert qt < most and 0.75 * SMS <= items <= SMS


@pytest.mark.parametrize("E,n,Hq,Hkv", [(1, 30, 16, 16), (1, 77, 16, 4), (1, 2000, 16, 16), (4, 200, 16, 2), (16, 64, 16, 4), (64, 32, 16, 2), (16, 2048, 16, 4),
                                        (2048, 4, 16, 4), (512, 16, 16, 16), (3, 50, 256, 1), (3, 50, 300, 300)])
def test_long_portions_and_full_chips_keep_full_tiles(E, n, Hq, Hkv):
    qt, most, _ = _items(E * n, E, Hq, Hkv)
    assert qt == most


def test_bounds_hold_everywhere():
    r = random.Random(0)
    for _ in range(3000):
        Hkv = r.choice([1, 2, 4, 8, 16, 37, 200])
        Hq = Hkv * r.choice([1, 2, 3, 5, 8, 16, 128])
        E = r.randint(1, 600)
        T = E + r.randint(0, 1 << r.randint(0, 22))
        qt, most, items = _items(T, E, Hq, Hkv)
        assert 1 <= qt <= most and (qt == most or items <= SMS)
