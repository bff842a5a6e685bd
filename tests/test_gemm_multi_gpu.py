"""Several narrow products in one launch against float64: results that end inside tiles, both forms of the first operand, results written across, ranges of unequal
length, and the number of ranges that is chosen."""
import pytest
import torch

from nanorlhf_b200 import _C

FITS = [0, 148, 74, 45, 33, 26, 22, 15, 15]


@pytest.mark.parametrize("tiles,blocks,ranges", [
    ([12, 12], [104, 104], 5), ([12, 2, 2, 36], [104] * 4, 2), ([70, 70, 24, 12, 70], [104] * 5, 1), ([52, 52, 52], [24, 4, 4], 1), ([1], [3], 1), ([1, 1], [8, 64], 2),
])
def test_ranges(tiles, blocks, ranges):
    n = _C.gemm_tc_multi_splits(tiles, blocks, 148, FITS)
    assert n == ranges
    assert all(-(-b // -(-b // n)) == n for b in blocks)


def _run(shapes, a_mn, flips, splits, seed):
    from nanorlhf_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    a = [f(K, M) if a_mn else f(M, K) for M, N, K in shapes]
    wide = [f(K, N + 16) for M, N, K in shapes]
    b = [w[:, 8:8 + N] for w, (M, N, K) in zip(wide, shapes)]                # rows of their own stride
    out = [torch.full((N, M) if t else (M, N), 7.0, device="cuda", dtype=torch.bfloat16) for t, (M, N, K) in zip(flips, shapes)]
    alpha = [0.5 * (i + 1) for i in range(len(shapes))]
    native.ext().gemm_tc_multi(a, b, out, flips, alpha, a_mn, splits)
    for x, y, o, t, al, (M, N, K) in zip(a, b, out, flips, alpha, shapes):
        xd = x.double().T if a_mn else x.double()
        want, mag = al * (xd @ y.double()), al * (xd.abs() @ y.double().abs())
        got = o.double().T if t else o.double()
        # one rounding to bf16 and float sums of K products, cut off at 2^-23 of a partial sum every 16 products
        assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + (K / 16 + 8) * 2.0 ** -23 * mag).all()


@pytest.mark.gpu
@pytest.mark.parametrize("splits", [0, 1, 2, 4, 7])
@pytest.mark.parametrize("K", [1800, 2696])
def test_token_contractions(splits, K):
    if splits > 0 and -(-(-(-K // 64)) // -(-(-(-K // 64)) // splits)) != splits:
        pytest.skip("an empty range")
    _run([(8, 8, K), (136, 64, K), (256, 72, K), (264, 192, K), (1544, 16, K), (64, 64, K)], True, [False, True, False, True, True, False], splits, K)


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 129, 700])
@pytest.mark.parametrize("splits", [0, 1, 2])
def test_row_major_operands_with_contractions_of_their_own(M, splits):
    _run([(M, 64, 1536), (M, 8, 264), (M, 64, 520)], False, [False] * 3, splits, M)


@pytest.mark.gpu
@pytest.mark.parametrize("r,r_down", [(64, 64), (72, 72), (64, 72), (72, 64)])
def test_groups_of_either_rank(r, r_down):
    from nanorlhf_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(r + r_down)
    f = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()  # noqa: E731
    T, n = 300, 7                                                            # more products than one launch takes
    gs, x, t, ws, Bs, a = [f(T, 136) for _ in range(n)], f(T, 128), f(T, n * r), [f(136, 128) for _ in range(n)], [f(136, r) for _ in range(n)], f(n * r, 128)
    more = (f(T, 264), f(T, r_down))
    gx, ga, gbs, (gb_more, ga_more) = gemm._group_backward(gs, x, t, a, ws, Bs, 0.5, False, [more], [(more[1], x)])
    tp = torch.cat([0.5 * (y.double() @ B.double()) for y, B in zip(gs, Bs)], 1)
    tp_err = 2.0 ** -8 * tp.abs() + (136 / 16 + 8) * 2.0 ** -23 * torch.cat([0.5 * (y.double().abs() @ B.double().abs()) for y, B in zip(gs, Bs)], 1)
    near = lambda got, p, q, err=0.0: bool(((got.double() - p.T @ q).abs() <= 2.0 ** -8 * (p.T @ q).abs() + (1 + 2.0 ** -8) * err  # noqa: E731
                                            + (T / 16 + 8) * 2.0 ** -22 * (p.abs().T @ q.abs())).all())
    assert gx is None
    assert near(ga, tp, x.double(), tp_err.T @ x.double().abs())
    for i in range(n):
        assert near(gbs[i], gs[i].double(), t[:, i * r:(i + 1) * r].double())
    assert near(gb_more, more[0].double(), more[1].double()) and near(ga_more, more[1].double(), x.double())
