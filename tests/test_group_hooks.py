"""Projections that share their input go through a group's launch only where nothing else hangs on their calls."""
import pytest
import torch

from nanorlhf_b200 import ops
from nanorlhf_b200.models.lora import LoraLinear, lora_group_forward
from nanorlhf_b200.models.qwen2 import Linear


def _layers(n=3):
    g = torch.Generator().manual_seed(0)
    mods = [LoraLinear(Linear(16, 8), 8, 16) for _ in range(n)]
    with torch.no_grad():
        for m in mods:
            for p in m.parameters():
                p.copy_(torch.randn(p.shape, generator=g))
    return mods, torch.randn(5, 16, generator=g)


def test_plain_adapters_are_a_group(monkeypatch):
    mods, x = _layers()
    groups, group = [], ops.lora_linear_group
    monkeypatch.setattr(ops, "lora_linear_group", lambda *a: groups.append(1) or group(*a))
    ys = lora_group_forward(x, mods)
    assert groups and all(torch.equal(y, m(x)) for y, m in zip(ys, mods))


@pytest.mark.parametrize("what", ["forward", "pre", "backward", "instance", "subclass"])
def test_what_hangs_on_one_of_them_runs(what):
    mods, x = _layers()
    x.requires_grad_()
    seen = []
    if what == "forward":
        mods[1].register_forward_hook(lambda m, a, y: 3 * y)
    elif what == "pre":
        mods[1].register_forward_pre_hook(lambda m, a: (2 * a[0],))
    elif what == "backward":
        mods[1].register_full_backward_hook(lambda *_: seen.append(1))
    elif what == "instance":
        mods[1].forward = lambda a: 5 * LoraLinear.forward(mods[1], a)
    else:
        class Halved(LoraLinear):
            def forward(self, a):
                return 0.5 * super().forward(a)
        mods[1].__class__ = Halved
    ys = lora_group_forward(x, mods)
    assert all(torch.equal(y, m(x)) for y, m in zip(ys, mods))
    if what == "backward":
        ys[1].sum().backward()
        assert seen


def test_hooks_of_the_reward_models_adapters_run(monkeypatch):
    from types import SimpleNamespace

    from nanorlhf_b200.models import deberta_v3
    from nanorlhf_b200.ops import native
    cfg = deberta_v3.DebertaV3Config.tiny()
    attn = deberta_v3.DisentangledSelfAttention(cfg)
    attn.query_proj = LoraLinear(attn.query_proj, 8, 16)
    attn.key_proj = LoraLinear(attn.key_proj, 8, 16)
    attn.value_proj = LoraLinear(attn.value_proj, 8, 16)
    monkeypatch.setattr(native, "ext", lambda: SimpleNamespace(attn_varlen_fwd=lambda q, *a: (q, None)))      # the attention itself runs on the GPU only
    x, rel = torch.randn(5, cfg.hidden_size), torch.randn(2 * attn.span, cfg.hidden_size)
    want = attn.forward_packed(x, None, 5, None, rel)
    attn.query_proj.register_forward_hook(lambda m, a, y: 3 * y)
    assert torch.equal(attn.forward_packed(x, None, 5, None, rel), 3 * want)
