"""The delta-rule scan that takes 32 tokens at a time on the tensor cores (csrc/delta_chunk_tc.cu) against the recurrence in float64."""
import pytest
import torch

from test_delta_blocked_gpu import _run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("news,olds,H,KH,D,Dv,gla,offset", [
    ([1], [0], 1, 1, 1, 1, False, 0),                                     # the smallest state
    ([32, 31, 33, 97], [0, 3, 7, 0], 4, 4, 128, 128, False, 0),           # edges of a chunk; fresh and carried
    ([5, 1, 64, 65], [0, 3, 7, 0], 4, 2, 64, 48, False, 0),               # shared key heads, 64-row form, ragged columns
    ([6, 70], [2, 0], 3, 3, 65, 129, False, 0),                           # rows just above the 64-row form, a column behind the first block's
    ([6, 40], [2, 0], 3, 1, 13, 7, False, 3),                             # unaligned vectors
    ([50, 4], [0, 3], 2, 1, 128, 300, True, 0),                           # accumulation without the delta
    ([300] * 20, [0, 5] * 10, 8, 8, 64, 64, True, 1),                     # more blocks than SMs
])
def test_chunked_scan_against_float64(news, olds, H, KH, D, Dv, gla, offset):
    got, want, s, want_s = _run(news, olds, H, KH, D, Dv, False, gla, offset, "chunked")
    # as for the form of four tokens: float32 sums, terms of a product below 2^-24 left out, sums of at most 64 products cut off at 2^-24 each
    assert ((got - want).norm() / want.norm()).item() < 1e-6
    assert ((s - want_s).norm() / want_s.norm()).item() < 1e-6


def test_auto_takes_it_for_portions_with_one_decay_per_head():
    a = _run([40, 33], [0, 3], 2, 2, 64, 64, False, False, 0, "auto")[0]
    assert torch.equal(a, _run([40, 33], [0, 3], 2, 2, 64, 64, False, False, 0, "chunked")[0])
    with pytest.raises(RuntimeError):
        _run([40], [0], 2, 2, 64, 64, True, False, 0, "chunked")


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_what_is_not_finite_stays_with_its_column_and_the_tokens_behind(value):
    from nanorlhf_b200 import _C
    from nanorlhf_b200.ops import hybrid as hy
    from nanorlhf_b200.sampler.hybrid_sampler import StepPlan
    H, D, T = 1, 64, 80
    g = torch.Generator(device="cuda").manual_seed(3)
    sched = _C.StepScheduler(16, 16, 1)
    data, E, _, MB = sched.plan([sched.open()], [T])
    plan = StepPlan(torch.from_numpy(data).to("cuda"), E, T, MB)
    qkv = torch.randn(T, 3 * D, generator=g, device="cuda") * 0.1
    beta, decay = torch.full((T, H), 0.5, device="cuda"), torch.full((T, H), 0.9, device="cuda")

    def run(x):
        o, state = torch.empty(T, D, device="cuda"), torch.zeros(1, H, D, D, device="cuda")
        hy.delta_scan(x, D, 2 * D, beta, decay, state, o, plan, H, False, impl="chunked")
        return o
    want, bad = run(qkv), qkv.clone()
    bad[41, 2 * D + 7] = value                           # one value vector's element, in the middle of a chunk
    got = run(bad)
    spoilt = torch.zeros(T, D, dtype=torch.bool, device="cuda")
    spoilt[41:, 7] = True
    assert torch.equal(torch.isfinite(got), ~spoilt)
    assert torch.equal(got[~spoilt], want[~spoilt])
