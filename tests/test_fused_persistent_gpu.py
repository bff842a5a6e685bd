"""The training step's fused GEMMs and the projections of one input where a pair of blocks goes through several tiles: both accumulators in turn, tiles and chunks that are skipped
between full ones, slabs that are written again while their last contents leave, and the switch from one product to another inside a block."""
import pytest
import torch

pytestmark = pytest.mark.gpu

HALF, SUM = 2.0 ** -8, 2.0 ** -20            # roundings to bf16, float sums of at most 600 products relative to the sum of their magnitudes


def _r(g, *shape, std=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * std).bfloat16()


def _pairs():
    return torch.cuda.get_device_properties(0).multi_processor_count // 2


# the last column tile has one, two or three of its four chunks, the last row tile one warp's rows or all but some
@pytest.mark.parametrize("M,F,K,r", [(2600, 5192, 72, 8), (2049, 5128, 64, 16), (1300, 16 * 641, 136, 8), (5150, 2688, 8, 64)])
def test_gate_up_and_their_gradients(M, F, K, r):
    from nanorlhf_b200.ops import native
    ext, g = native.ext(), torch.Generator(device="cuda").manual_seed(M + F)
    assert -(-M // 256) * -(-F // 256) > 2 * _pairs()
    x, wg, wu, t, bg, bu = _r(g, M, K), _r(g, F, K, std=K ** -0.5), _r(g, F, K, std=K ** -0.5), _r(g, M, 2 * r), _r(g, F, r, std=0.1), _r(g, F, r, std=0.1)
    act, gate, up = ext.gemm_tc_swiglu_pair_keep(x, wg, wu, t[:, :r], t[:, r:], bg, bu)
    for y, w, tt, b in ((gate, wg, t[:, :r], bg), (up, wu, t[:, r:], bu)):
        ref, mag = x.double() @ w.double().T + tt.double() @ b.double().T, x.double().abs() @ w.double().abs().T + tt.double().abs() @ b.double().abs().T
        assert ((y.double() - ref).abs() <= HALF * 1.01 * ref.abs() + SUM * mag).all()
    assert torch.equal(act, ext.gemm_tc_swiglu_pair(x, wg, wu, t[:, :r], t[:, r:], bg, bu))
    ref = torch.nn.functional.silu(gate.double()) * up.double()
    assert ((act.double() - ref).abs() <= HALF * 1.01 * ref.abs() + 1e-30).all()
    del ref, mag
    w, a = _r(g, K, F, std=K ** -0.5), _r(g, r, F, std=0.1)
    t = t[:, :r]
    dg, du = ext.gemm_tc_dswiglu(x, w, t, a, gate, up)
    d, mag = x.double() @ w.double() + t.double() @ a.double(), x.double().abs() @ w.double().abs() + t.double().abs() @ a.double().abs()
    gd, ud, s = gate.double(), up.double(), torch.sigmoid(gate.double())
    for got, f in ((dg, ud * (s + gd * s * (1 - s))), (du, gd * s)):
        err = 2.02 * HALF * (d * f).abs() + SUM * mag * f.abs() + 2.0 ** -20 * d.abs() * (ud.abs() + gd.abs()) * (1 + gd.abs())
        assert ((got.double() - d * f).abs() <= err + 1e-30).all()


@pytest.mark.parametrize("M,N,Ks", [(5200, 1544, (64, 200)), (20000, 520, (72, 8, 136, 64)), (9473, 3080, (8, 72, 64))])
def test_sums_of_products(M, N, Ks):
    from nanorlhf_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(M)
    assert -(-M // 256) * -(-N // 256) > _pairs()
    a, b = [_r(g, M, k) for k in Ks], [_r(g, k, N) for k in Ks]
    ref = sum(x.double() @ y.double() for x, y in zip(a, b))
    mag = sum(x.double().abs() @ y.double().abs() for x, y in zip(a, b))
    assert ((native.ext().gemm_tc_sum(a, b).double() - ref).abs() <= HALF * 1.01 * ref.abs() + SUM * mag).all()


@pytest.mark.parametrize("M", [5000, 9473])
@pytest.mark.parametrize("Ns,r,biases", [((1536, 256, 264), 16, (True, False, True)), ((520, 8, 1024, 200), 0, (False, True, True, False)), ((72, 3080), 8, (True, True))])
@pytest.mark.parametrize("cg,bn", [(0, 0), (1, 64), (1, 128), (2, 128), (2, 192), (2, 256)])
def test_projections_of_one_input(M, Ns, r, biases, cg, bn):
    from nanorlhf_b200.ops import gemm, native
    g, K = torch.Generator(device="cuda").manual_seed(M + sum(Ns)), 136
    assert bn == 0 or -(-M // (128 * cg)) * sum(-(-n // bn) for n in Ns) > 2 * _pairs() // cg
    x, ws, bs = _r(g, M, K), [_r(g, n, K) for n in Ns], [_r(g, n) if b else None for n, b in zip(Ns, biases)]
    t, Bs = _r(g, M, max(1, len(Ns) * r)), [_r(g, n, r) for n in Ns]
    ts = [t[:, i * r:(i + 1) * r] for i in range(len(Ns))] if r else []
    got = native.ext().gemm_tc_cat(x, ws, bs, ts, Bs if r else [], cg, bn)
    for i in range(len(Ns)):
        assert torch.equal(got[i], gemm.gemm(x, ws[i], a2=ts[i] if r else None, b2=Bs[i] if r else None, bias=bs[i], split_k=0))


@pytest.mark.parametrize("M,N,K", [(5200, 1544, 136), (9473, 520, 72), (2600, 5192, 64)])
def test_residuals(M, N, K):
    from nanorlhf_b200.ops import gemm
    g = torch.Generator(device="cuda").manual_seed(N)
    x, w, res = _r(g, M, K), _r(g, N, K), _r(g, M, N + 8)[:, :N]
    assert torch.equal(gemm.gemm(x, w, residual=res), res + gemm.gemm(x, w, split_k=0))


@pytest.mark.parametrize("M,V", [(1500, 8200), (3000, 16392)])
def test_log_probabilities_of_several_ranges_a_pair(M, V):
    from nanorlhf_b200.ops import native
    ext, g = native.ext(), torch.Generator(device="cuda").manual_seed(M)
    h, w, t = _r(g, M, 72), _r(g, V, 72, std=0.3), torch.randint(0, V, (M,), generator=g, device="cuda").int()
    splits = 2 * _pairs() // -(-M // 256) + 3                              # more items than pairs
    z = torch.empty(M, V, device="cuda")
    lp, ent, lse = ext.lmhead_logprob_fwd(h, w, t, 1.0, splits, z)
    zd = h.double() @ w.double().T
    assert ((z.double() - zd).abs() <= 16 * 2.0 ** -23 * (h.double().abs() @ w.double().abs().T)).all()
    ref = torch.log_softmax(zd, -1)
    # logarithms of about 20 from sums of thousands of float exponentials of approximate 2^x (2^-21 each, relative): 20 times 2^-18
    assert (lp.double() - ref.gather(1, t.long()[:, None])[:, 0]).abs().max() <= 1e-4
    assert (ent.double() + (ref.exp() * ref).sum(-1)).abs().max() <= 1e-4 and (lse.double() - torch.logsumexp(zd, -1)).abs().max() <= 1e-4
