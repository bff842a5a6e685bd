"""Which kernel a step of the paged attention takes, and what the tcgen05 form leaves alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _step(news, olds, H, Hkv, D=128, seed=0):
    from nanorlhf_b200 import _C
    from nanorlhf_b200.sampler.hybrid_sampler import StepPlan
    g = torch.Generator(device="cuda").manual_seed(seed)
    pages = sum((o + n + 15) // 16 for o, n in zip(olds, news)) + 4
    sched = _C.StepScheduler(pages, 16, len(news))
    sids = [sched.open() for _ in news]
    if any(olds):
        sched.plan([s for s, o in zip(sids, olds) if o], [o for o in olds if o])
    data, E, T, MB = sched.plan(sids, list(news))
    kc, vc = (torch.randn(pages, Hkv, 16, D, generator=g, device="cuda").bfloat16() for _ in range(2))
    q = torch.randn(T, H * D, generator=g, device="cuda").bfloat16().float()
    return StepPlan(torch.from_numpy(data).cuda(), E, T, MB), kc, vc, q


def _run(step, impl, out=None, **kw):
    from nanorlhf_b200.ops import hybrid as hy
    plan, kc, vc, q = step
    out = torch.empty(q.shape, device="cuda", dtype=torch.bfloat16) if out is None else out
    hy.window_attention(q, kc, vc, plan, 1 << 30, kc.shape[-1] ** -0.5, 1.0, out, impl=impl, **kw)
    return out


def test_refused_forms_stay_on_the_general_kernel():
    step = _step([90, 40], [0, 30], 8, 2)
    slope = torch.rand(8, device="cuda")
    odd = torch.empty(130, 8 * 128 + 8, device="cuda", dtype=torch.bfloat16)[:, :8 * 128]          # rows of the result not 32-byte aligned
    for kw in ({"head_slope": slope}, {"head_scale": slope}, {"dist_bias": torch.randn(5, 8, device="cuda")}, {"out": odd}):
        with pytest.raises(RuntimeError):
            _run(step, "tc", **kw)
        assert torch.equal(_run(step, "auto", **kw), _run(step, "mma", **{k: v if k != "out" else torch.empty_like(v) for k, v in kw.items()}))
    small = _step([90, 40], [0, 30], 8, 2, D=64)
    with pytest.raises(RuntimeError):
        _run(small, "tc")
    assert torch.equal(_run(small, "auto"), _run(small, "mma"))


@pytest.mark.parametrize("H,Hkv", [(16, 16), (8, 2), (3, 1), (128, 1)])
@pytest.mark.parametrize("news,olds", [([4] * 64, [0] * 64), ([2] * 40 + [70], [100] * 40 + [0]), ([7] * 33, [13] * 33), ([1] * 90 + [5], [300] * 91)])
def test_rows_do_not_depend_on_how_a_step_is_cut(H, Hkv, news, olds):
    step = _step(news, olds, H, Hkv)
    plan, kc, vc, q = step
    got, t0 = _run(step, "tc"), 0
    assert ((got.float() - _run(step, "mma").float()).norm() / got.float().norm()).item() < 6e-3
    for e in (0, len(news) // 2, len(news) - 1):                # entries alone: full tiles of one run
        t0, n = sum(news[:e]), news[e]
        alone = _step([n], [olds[e]], H, Hkv)[0]
        alone.block_table[0, :plan.block_table.shape[1]] = plan.block_table[e, :alone.block_table.shape[1]]
        assert torch.equal(_run((alone, kc, vc, q[t0:t0 + n]), "tc"), got[t0:t0 + n])
