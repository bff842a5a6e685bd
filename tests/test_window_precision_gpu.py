"""The tcgen05 prompt attention is as near to float64 as the mma.sync form, where single weights make up most of a row as well."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sharp", [1.0, 4.0, 16.0])          # standard deviation of the scores: flat rows, a few weights, one weight
@pytest.mark.parametrize("f32", [False, True])
def test_no_further_from_float64_than_the_mma_form(sharp, f32):
    from test_window_tc_gpu import D
    from test_window_routes_gpu import _run, _step
    plan, kc, vc, q = _step([900, 300], [0, 500], 8, 2, seed=3)
    q = (q * sharp).bfloat16().float()
    err = {}
    for impl in ("mma", "tc"):
        out = torch.empty(q.shape, device="cuda", dtype=torch.float32 if f32 else torch.bfloat16)
        _run((plan, kc, vc, q), impl, out=out)
        worst, total, t0 = 0.0, 0.0, 0
        for e, (n, old) in enumerate([(900, 0), (300, 500)]):
            L = n + old
            pg = plan.block_table[e, :(L + 15) // 16].long().repeat_interleave(16)[:L]
            at = torch.arange(L, device="cuda")
            seen = at <= torch.arange(old, L, device="cuda")[:, None]
            for h in range(8):
                k, v = (c[pg, h // 4, at % 16].double() for c in (kc, vc))
                s = (q[t0:t0 + n, h * D:(h + 1) * D].double() @ k.T * D ** -0.5).masked_fill(~seen, -torch.inf)
                want = s.softmax(-1) @ v
                worst += (out[t0:t0 + n, h * D:(h + 1) * D].double() - want).square().sum().item()
                total += want.square().sum().item()
            t0 += n
        err[impl] = (worst / total) ** 0.5
    # both round each weight once (2^-9); what differs is how often a row's largest weight is rounded at all: 2 % for the blocks' sizes
    assert err["tc"] < 1.02 * err["mma"], err
