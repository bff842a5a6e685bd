"""The delta-rule scan that takes four tokens at a time (csrc/recurrent.cu) against the recurrence in float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(news, olds, H, KH, D, Dv, per_channel, gla, offset, impl):
    from nanorlhf_b200 import _C
    from nanorlhf_b200.ops import hybrid as hy
    from nanorlhf_b200.sampler.hybrid_sampler import StepPlan
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(D * 7 + Dv)

    def f(*s):
        return torch.randn(*s, generator=g, device=dev)
    sched = _C.StepScheduler(sum((o + n + 15) // 16 for o, n in zip(olds, news)) + 4, 16, len(news))
    sids = [sched.open() for _ in news]
    if any(olds):
        sched.plan([s for s, o in zip(sids, olds) if o], [o for o in olds if o])
    data, E, T, MB = sched.plan(sids, list(news))
    plan = StepPlan(torch.from_numpy(data).to(dev), E, T, MB)
    q, k = (torch.nn.functional.normalize(f(T, KH, D), dim=-1) for _ in range(2))
    v = f(T, H, Dv)
    qkv = torch.cat([f(T, offset), q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], 1).contiguous()[:, offset:]
    beta = None if gla else torch.sigmoid(f(T, H))
    decay = torch.exp(-torch.nn.functional.softplus(f(T, H * D if per_channel else H) - 3))
    decay[0], decay[-1] = 0.0, 1.0
    state = f(len(news), H, D, Dv) * 0.3
    want_s, want = state.double(), torch.empty(T, H, Dv, device=dev, dtype=torch.float64)
    cu = plan.cu.tolist()
    for e in range(E):
        slot = int(plan.state_slot[e])
        S = want_s[slot] if olds[e] else torch.zeros_like(want_s[slot])
        for t in range(cu[e], cu[e + 1]):
            kt, qt = (x[t].double().repeat_interleave(H // KH, 0)[:, :, None] for x in (k, q))
            S = S * decay[t].double().view(H, -1, 1)
            u = v[t].double() if gla else beta[t].double()[:, None] * (v[t].double() - (S * kt).sum(1))
            S = S + kt * u[:, None]
            want[t] = (S * qt).sum(1)
        want_s[slot] = S
    o = torch.full((T, H * Dv), 9.0, device=dev)
    hy.delta_scan(qkv, KH * D, 2 * KH * D, beta, decay, state, o, plan, KH, per_channel, impl=impl)
    return o.double(), want.reshape(T, -1), state.double(), want_s


@pytest.mark.parametrize("news,olds,H,KH,D,Dv,per_channel,gla,offset", [
    ([1], [0], 1, 1, 1, 1, False, False, 0),                              # the smallest state
    ([4, 3, 5, 41], [0, 3, 7, 0], 4, 4, 128, 128, False, False, 0),       # edges of a chunk; fresh and carried
    ([5, 1, 9, 60], [0, 3, 7, 0], 4, 2, 128, 128, True, False, 0),        # shared key heads, decay per channel
    ([5, 1, 9, 60], [0, 3, 7, 0], 4, 2, 64, 48, True, False, 0),          # 64-row form, ragged columns
    ([6, 30], [2, 0], 3, 3, 65, 72, False, False, 0),                     # rows just above the 64-row form
    ([6, 30], [2, 0], 3, 1, 13, 7, True, False, 3),                       # unaligned vectors
    ([50, 4], [0, 3], 2, 1, 128, 300, True, True, 0),                     # accumulation without the delta, many columns
    ([13] * 40, [0, 5] * 20, 8, 8, 64, 64, False, False, 0),              # eight columns per thread (enough blocks)
])
def test_blocked_scan_against_float64(news, olds, H, KH, D, Dv, per_channel, gla, offset):
    got, want, s, want_s = _run(news, olds, H, KH, D, Dv, per_channel, gla, offset, "blocked")
    # float32 sums over <= 128 rows and <= 60 tokens of unit keys: a few 2^-24 relative to the result's norm
    assert ((got - want).norm() / want.norm()).item() < 1e-6
    assert ((s - want_s).norm() / want_s.norm()).item() < 1e-6


def test_auto_takes_it_for_portions_only():
    a = _run([40, 33], [0, 3], 2, 2, 64, 64, True, False, 0, "auto")[0]
    assert torch.equal(a, _run([40, 33], [0, 3], 2, 2, 64, 64, True, False, 0, "blocked")[0])
    a = _run([2, 1], [0, 3], 2, 2, 64, 64, True, False, 0, "auto")[0]
    assert torch.equal(a, _run([2, 1], [0, 3], 2, 2, 64, 64, True, False, 0, "column")[0])
