"""The chunked delta-rule scan whose blocks share the chunks of all items: bit for bit what blocks with one item each give, and when it is taken."""
import pytest
import torch

from nanorlhf_b200 import _C

SMS = 148


@pytest.mark.parametrize("E,T,heads,Dv,shared", [
    (10, 10 * 2048, 16, 128, True), (12, 12 * 700, 16, 128, True), (11, 11 * 300, 16, 64, True), (16, 16 * 2048, 16, 128, False), (9, 9 * 2048, 16, 128, False),
    (32, 32 * 1000, 16, 128, False), (16, 16 * 256, 16, 128, False), (5, 5 * 2048, 16, 256, True), (1, 2048, 149, 128, True), (10, 10 * 32, 16, 128, False),
])
def test_rule(E, T, heads, Dv, shared):
    assert bool(_C.delta_scan_shared(E, T, heads, Dv, SMS)) == shared


def _inputs(news, olds, H, KH, D, Dv, gla, seed):
    from nanorlhf_b200.sampler.hybrid_sampler import StepPlan
    g = torch.Generator(device="cuda").manual_seed(seed)
    f = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    sched = _C.StepScheduler(sum((o + n + 15) // 16 for o, n in zip(olds, news)) + 4, 16, len(news))
    sids = [sched.open() for _ in news]
    if any(olds):
        sched.plan([s for s, o in zip(sids, olds) if o], [o for o in olds if o])
    data, E, T, MB = sched.plan(sids, list(news))
    q, k = (torch.nn.functional.normalize(f(T, KH, D), dim=-1) for _ in range(2))
    qkv = torch.cat([q.reshape(T, -1), k.reshape(T, -1), f(T, H * Dv)], 1).contiguous()
    beta = None if gla else torch.sigmoid(f(T, H))
    decay = torch.exp(-torch.nn.functional.softplus(f(T, H) - 3))
    return StepPlan(torch.from_numpy(data).to("cuda"), E, T, MB), qkv, beta, decay, f(len(news), H, D, Dv) * 0.3


@pytest.mark.gpu
@pytest.mark.parametrize("news,olds,H,KH,D,Dv,gla", [
    ([400] * 10, [0, 5] * 5, 16, 16, 128, 128, False),                     # a little more than a round; items cut nearly everywhere
    ([700] + [33] * 9 + [350] * 10, [0] * 20, 8, 4, 64, 64, False),        # one long entry sets the share: some blocks have no work
    ([500, 470, 1, 32, 512, 300, 200, 410, 600, 650, 620], [0, 3, 0, 9, 0, 2, 0, 0, 1, 0, 0], 15, 5, 64, 64, False),      # portions of one token and one chunk
    ([900] * 5, [0, 3, 0, 7, 0], 16, 16, 128, 200, True),                  # two blocks of columns, the second ragged; accumulation
])
def test_the_bits_of_whole_items(news, olds, H, KH, D, Dv, gla):
    from nanorlhf_b200.ops import hybrid as hy
    assert _C.delta_scan_shared(len(news), sum(news), H, Dv, SMS)
    plan, qkv, beta, decay, state = _inputs(news, olds, H, KH, D, Dv, gla, len(news) + D)
    o, s = torch.empty(sum(news), H * Dv, device="cuda"), state.clone()
    hy.delta_scan(qkv, KH * D, 2 * KH * D, beta, decay, s, o, plan, KH, False, impl="chunked")
    # entry by entry there are fewer items than SMs
    o1, s1, cu = torch.empty_like(o), state.clone(), plan.cu.tolist()
    for e in range(len(news)):
        r = slice(cu[e], cu[e + 1])
        _C.delta_scan(qkv[r], KH * D, 2 * KH * D, None if beta is None else beta[r].contiguous(), decay[r].contiguous(), s1, o1[r],
                      torch.tensor([0, news[e]], dtype=torch.int32, device="cuda"), plan.start[e:e + 1].contiguous(), plan.state_slot[e:e + 1].contiguous(),
                      KH, False, 5)
    assert torch.equal(o, o1) and torch.equal(s, s1)
