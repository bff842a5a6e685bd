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
