"""Projections of one input in one launch: the bits of their own GEMMs, on every tile, with results that end inside tiles, with and without second operands and biases."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _r(g, *s):
    return torch.randn(*s, generator=g, device="cuda").bfloat16()


@pytest.mark.parametrize("M", [1, 129, 300])
@pytest.mark.parametrize("Ns", [(8,), (264, 8, 256), (128, 200), (72, 64, 520, 8)])
@pytest.mark.parametrize("r,biases", [(0, (True, False, True, True)), (16, (False, True, False, False))])
@pytest.mark.parametrize("cg,bn", [(0, 0), (1, 64), (1, 128), (2, 128), (2, 192), (2, 256)])
def test_the_bits_of_their_own_gemms(M, Ns, r, biases, cg, bn):
    from nanorlhf_b200.ops import gemm, native
    g = torch.Generator(device="cuda").manual_seed(M + sum(Ns) + r)
    K = 136
    x, ws, bs = _r(g, M, K + 8)[:, :K], [_r(g, N, K) for N in Ns], [_r(g, N) if b else None for N, b in zip(Ns, biases)]
    t, Bs = _r(g, M, max(1, len(Ns) * r)), [_r(g, N, r) for N in Ns]
    ts = [t[:, i * r:(i + 1) * r] for i in range(len(Ns))] if r else []
    got = native.ext().gemm_tc_cat(x, ws, bs, ts, Bs if r else [], cg, bn)
    for i, N in enumerate(Ns):
        want = gemm.gemm(x, ws[i], a2=ts[i] if r else None, b2=Bs[i] if r else None, bias=bs[i], split_k=0)
        assert got[i].shape == (M, N) and torch.equal(got[i], want)


def test_cut_contractions_keep_their_own_launches():
    from nanorlhf_b200.ops import gemm, native
    g = torch.Generator(device="cuda").manual_seed(0)
    x, ws = _r(g, 128, 4096), [_r(g, 256, 4096), _r(g, 64, 4096)]
    assert native.ext().gemm_tc_auto_splits(128, 256, 4096) > 1 and gemm.linears(x, ws, [None, None]) is None
    assert gemm.linears(x[:0], ws, [None, None]) is None
