"""Fused kernels stand in for a module's call only where that call runs the module's own forward and nothing else."""
import pytest
import torch
import torch.nn as nn

from nanorlhf_b200.models.lora import LoraLinear, plain_module
from nanorlhf_b200.models.qwen2 import Linear, RMSNorm


def _modules():
    return [(Linear(8, 8, bias=False), Linear), (RMSNorm(8, 1e-6), RMSNorm), (LoraLinear(Linear(8, 8, bias=False), 8, 16), LoraLinear)]


@pytest.mark.parametrize("i", range(3))
def test_plain_modules_and_what_makes_them_otherwise(i, monkeypatch):
    m, cls = _modules()[i]
    assert plain_module(m, cls)
    m.forward = lambda x: x                                         # as hook libraries do
    assert not plain_module(m, cls)
    del m.forward
    for register in (m.register_forward_hook, m.register_forward_pre_hook, m.register_full_backward_hook):
        handle = register(lambda *_: None)
        assert not plain_module(m, cls)
        handle.remove()
    for register in (nn.modules.module.register_module_forward_hook, nn.modules.module.register_module_forward_pre_hook):
        handle = register(lambda *_: None)
        try:
            assert not plain_module(m, cls)
        finally:
            handle.remove()
    assert plain_module(m, cls)
    monkeypatch.setattr(cls, "forward", lambda self, x: x)          # the class's forward replaced
    assert not plain_module(m, cls)


def test_subclasses_with_a_forward_or_call_of_their_own():
    class Doubled(Linear):
        def forward(self, x):
            return 2 * super().forward(x)

    class Counted(Linear):
        def __call__(self, x):
            return super().__call__(x)

    class Named(Linear):
        pass
    assert [plain_module(c(8, 8, bias=False), Linear) for c in (Doubled, Counted, Named)] == [False, False, True]
    assert not plain_module(nn.Linear(8, 8), Linear)
