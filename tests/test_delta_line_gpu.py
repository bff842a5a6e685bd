"""The chunked delta-rule scan whose blocks share the chunks of all items: bit for bit what blocks with one item each give, when it comes into question by the number of
items, and when the lengths say that it pays."""
import heapq
import random

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
    plan, qkv, beta, decay, state = _inputs(news, olds, H, KH, D, Dv, gla, len(news) + D)
    o, s = torch.empty(sum(news), H * Dv, device="cuda"), state.clone()
    hy.delta_scan(qkv, KH * D, 2 * KH * D, beta, decay, s, o, plan, KH, False, impl="line")
    for plan.lengths in (None, news):                                      # as the lengths say, found by the GPU or by the host
        o0, s0 = torch.empty_like(o), state.clone()
        hy.delta_scan(qkv, KH * D, 2 * KH * D, beta, decay, s0, o0, plan, KH, False, impl="chunked")
        assert torch.equal(o, o0) and torch.equal(s, s0)
    # entry by entry there are fewer items than SMs
    o1, s1, cu = torch.empty_like(o), state.clone(), plan.cu.tolist()
    for e in range(len(news)):
        r = slice(cu[e], cu[e + 1])
        _C.delta_scan(qkv[r], KH * D, 2 * KH * D, None if beta is None else beta[r].contiguous(), decay[r].contiguous(), s1, o1[r],
                      torch.tensor([0, news[e]], dtype=torch.int32, device="cuda"), plan.start[e:e + 1].contiguous(), plan.state_slot[e:e + 1].contiguous(),
                      KH, False, 5)
    assert torch.equal(o, o1) and torch.equal(s, s1)


def test_hosts_with_the_lengths_decide_without_the_gpu():
    assert _C.delta_line_pays([2048] * 10, 16, 128, SMS) and not _C.delta_line_pays([4000] + [400] * 9, 16, 128, SMS)
    rng = random.Random(1)
    for _ in range(300):
        news, heads = [rng.randint(0, 2000) for _ in range(rng.randint(1, 40))], rng.choice([4, 16, 40])
        if _C.delta_line_pays(news, heads, 128, SMS):
            chunks = _chunks(news)
            assert 1.13 * max(max(chunks), -(-sum(chunks) * heads // SMS)) + 4 < 0.9 * _whole(chunks, heads, SMS)


def _chunks(news):
    return [max(1, -(-n // 32)) for n in news]


def _cu(news):
    return torch.tensor([0, *torch.tensor(news).cumsum(0).tolist()], dtype=torch.int32, device="cuda")


def _whole(chunks, items, sms):
    """chunks in a row when whole items go to the SM that is free first"""
    free = [0] * sms
    for n in chunks:
        for _ in range(items):
            heapq.heappush(free, heapq.heappop(free) + n)
    return max(free)


@pytest.mark.gpu
@pytest.mark.parametrize("news,heads,Dv,taken", [
    ([2048] * 10, 16, 128, True), ([700] * 12, 16, 128, True), ([300] * 11, 16, 64, True), ([900] * 5, 16, 200, True), ([2048] * 16, 16, 128, False),
    ([4000] + [400] * 9, 16, 128, False), ([700] + [33] * 9 + [350] * 10, 8, 64, False),      # by the mean length they were taken, and slower for it
])
def test_lengths_decide(news, heads, Dv, taken):
    assert bool(_C.delta_line_plan(_cu(news), heads, Dv, SMS)[0]) == taken == _C.delta_line_pays(news, heads, Dv, SMS)


@pytest.mark.gpu
def test_never_taken_where_whole_items_are_as_fast():
    rng, taken = random.Random(4), 0
    for i in range(300):
        heads, E, lo = rng.choice([4, 8, 16, 32]), rng.randint(2, 60), rng.choice([30, 300, 900])
        news = [int(lo * (2000 / lo) ** rng.random()) if i % 2 else rng.randint(900, 1000) for _ in range(E)]
        chunks = _chunks(news)
        pays = _C.delta_line_pays(news, heads, 128, SMS)
        assert bool(_C.delta_line_plan(_cu(news), heads, 128, SMS)[0]) == pays
        if pays:
            taken += 1
            line = max(max(chunks), -(-sum(chunks) * heads // SMS))
            assert 1.13 * line + 4 < 0.9 * _whole(chunks, heads, SMS)
    assert taken >= 10


@pytest.mark.gpu
@pytest.mark.parametrize("news,heads,Dv,blocks", [([400] * 10, 16, 128, 148), ([700] + [33] * 9 + [0, 350, 1] * 5, 8, 300, 148), ([5, 90], 3, 64, 7), ([64] * 40, 4, 128, 13)])
def test_every_chunk_lies_in_one_segment(news, heads, Dv, blocks):
    taken, ends, segments = _C.delta_line_plan(_cu(news), heads, Dv, blocks, True)
    assert taken
    ends, segments, chunks, parts = ends.tolist(), segments.tolist(), _chunks(news), -(-Dv // 128)
    per, seen, cu = max(max(chunks), -(-sum(chunks) * heads * parts // blocks)), {}, _cu(news).tolist()
    for b in range(blocks):
        mine = segments[ends[0][b]:ends[1][b]]
        assert sum(s[1] for s in mine) <= per
        for i, (t0, n, t1, h, cb0, e, came, goes) in enumerate(mine):
            assert n > 0 and t1 == cu[e + 1] and (t0 - cu[e]) % 32 == 0
            assert not goes or i == 0                                    # what another block waits for is computed first
            assert not came or i == len(mine) - 1                        # what waits for another block is computed last
            if came:
                nxt = segments[ends[0][b + 1]]
                assert nxt[7] and nxt[3:6] == [h, cb0, e] and nxt[0] + 32 * nxt[1] == t0
            seen.setdefault((e, h, cb0), []).append(((t0 - cu[e]) // 32, n))
    assert len(seen) == len(news) * heads * parts
    for (e, _, _), runs in seen.items():
        runs.sort()
        assert runs[0][0] == 0 and all(a + n == b for (a, n), (b, _) in zip(runs, runs[1:])) and runs[-1][0] + runs[-1][1] == chunks[e]
