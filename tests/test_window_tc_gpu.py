"""The tcgen05 prompt-attention kernel over pages (csrc/attention_window_tc.cu) against a float64 softmax written out per entry."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
D = 128


def _run(news, olds, H, Hkv, window, softcap=0.0, chunked=False, keep=0, sink=False, gate=None, v_div=1, f32=False, impl="tc"):
    """(result, float64 oracle).  Page rows that no sequence holds are NaN: the kernel must not let them in."""
    from nanorlhf_b200 import _C
    from nanorlhf_b200.ops import hybrid as hy
    from nanorlhf_b200.sampler.hybrid_sampler import StepPlan
    dev = "cuda"
    g = torch.Generator(device=dev).manual_seed(len(news) * 1000 + H)
    pages = sum((o + n + 15) // 16 for o, n in zip(olds, news)) + 4
    sched = _C.StepScheduler(pages, 16, len(news))
    sids = [sched.open() for _ in news]
    if any(olds):
        sched.plan([s for s, o in zip(sids, olds) if o], [o for o in olds if o])
    data, E, T, MB = sched.plan(sids, list(news))
    plan = StepPlan(torch.from_numpy(data).to(dev), E, T, MB)
    kc = torch.full((pages, Hkv, 16, D), float("nan"), device=dev, dtype=torch.bfloat16)
    vc = torch.full((pages, Hkv // v_div, 16, D), float("nan"), device=dev, dtype=torch.bfloat16)
    q = (torch.randn(T, H * D, generator=g, device=dev) * 1.5).bfloat16().float()
    opt = {"head_sink": torch.randn(H, generator=g, device=dev)} if sink else {}
    if gate is not None:
        opt["gate"] = torch.randn(T, H if gate == "head" else H * D, generator=g, device=dev)
    want, t0 = torch.empty(T, H, D, device=dev, dtype=torch.float64), 0
    for e, (n, old) in enumerate(zip(news, olds)):
        L = n + old
        k, v = (torch.randn(L, h, D, generator=g, device=dev).bfloat16() for h in (Hkv, Hkv // v_div))
        pg = plan.block_table[e, :(L + 15) // 16].long().repeat_interleave(16)[:L]
        at = torch.arange(L, device=dev)
        kc[pg, :, at % 16], vc[pg, :, at % 16] = k, v
        p = torch.arange(old, L, device=dev)[:, None]
        first = p - p % window if chunked else p - window + 1
        seen = (at <= p) & ((at >= first) | ((at < keep) if not chunked else torch.zeros_like(at, dtype=torch.bool)))
        for h in range(H):
            kv = h // (H // Hkv)
            s = q[t0:t0 + n, h * D:(h + 1) * D].double() @ k[:, kv].double().T * D ** -0.5
            s = softcap * torch.tanh(s / softcap) if softcap else s
            s = s.masked_fill(~seen, -math.inf)
            if sink:
                s = torch.cat([s, opt["head_sink"][h].double().expand(n, 1)], 1)
            w = torch.softmax(s, -1)[:, :L]
            want[t0:t0 + n, h] = 0.7 * (w @ v[:, kv // v_div].double())
        t0 += n
    if gate is not None:
        want = want * torch.sigmoid(opt["gate"].double().view(T, H, -1))
    out = torch.empty(T, H * D, device=dev, dtype=torch.float32 if f32 else torch.bfloat16)
    hy.window_attention(q, kc, vc, plan, window, D ** -0.5, 0.7, out, impl=impl, softcap=softcap, chunked=chunked, keep_first=keep, v_div=v_div, **opt)
    return out.double(), want.reshape(T, -1)


@pytest.mark.parametrize("news,olds,H,Hkv,window,kw", [
    ([1], [0], 1, 1, 1, {}),                                              # the smallest call
    ([2, 1], [0, 0], 4, 4, 64, {}),
    ([128, 127, 129], [0, 0, 0], 4, 1, 1 << 30, {}),                      # edges of a key block; 32 tokens x 4 heads a tile
    ([300, 16, 17, 15], [0, 112, 111, 113], 6, 2, 128, {}),               # 42 tokens an item, 2 rows of a tile unused
    ([130, 257, 5, 1, 64, 31], [0, 100, 0, 500, 17, 3], 8, 2, 100, {}),   # several sequences in one item
    ([1] * 70 + [3], [50] * 71, 1, 1, 64, {}),                            # a run per token
    ([40, 9], [0, 300], 128, 1, 77, {}),                                  # one token a tile
    ([700, 33], [1000, 0], 8, 8, 256, {"softcap": 20.0}),
    ([700, 33], [1000, 0], 8, 1, 256, {"chunked": True, "sink": True, "gate": "head"}),
    ([700, 33], [1000, 0], 8, 2, 128, {"keep": 5, "gate": "cols"}),
    ([700, 33], [1000, 0], 8, 2, 128, {"keep": 200, "f32": True}),
    ([300, 33, 70], [1000, 0, 9], 8, 4, 300, {"v_div": 2, "f32": True}),
    ([1100] * 3, [0, 40, 1], 16, 4, 200, {}),                             # more items than SMs
])
def test_tc_kernel_against_softmax(news, olds, H, Hkv, window, kw):
    got, want = _run(news, olds, H, Hkv, window, **kw)
    # weights and result are rounded to bf16 (2^-9 each, relative); the sum over keys averages the first
    assert torch.isfinite(got).all() and ((got - want).norm() / want.norm()).item() < 6e-3
    assert ((got - want).abs().max() / want.abs().max()).item() < 2e-2


def test_auto_takes_the_kernel_and_refusals_stay():
    a, want = _run([90, 40], [0, 30], 8, 2, 64, impl="auto")
    b, _ = _run([90, 40], [0, 30], 8, 2, 64, impl="tc")
    assert torch.equal(a, b)
    c, _ = _run([90, 40], [0, 30], 8, 2, 64, impl="mma")
    assert not torch.equal(a, c) and ((a - c).norm() / want.norm()).item() < 6e-3
