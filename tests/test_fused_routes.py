"""Which calls of the MLP take the fused GEMM outside autograd; the kernel itself is put aside, so that the routes can be seen on the CPU."""
import pytest
import torch
import torch.nn as nn

from nanorlhf_b200 import ops
from nanorlhf_b200.models import lora
from nanorlhf_b200.models.qwen2 import Linear
from nanorlhf_b200.ops import gemm


@pytest.fixture
def fused(monkeypatch):
    monkeypatch.setattr(ops, "use_native", lambda t: True)
    monkeypatch.setattr(gemm, "swiglu_linears", lambda *a, **k: "fused")

    def call(gate, up, x=None):
        return lora.fused_swiglu_forward(torch.zeros(2, 8, dtype=torch.bfloat16) if x is None else x, gate, up)
    return call


def _pair(adapters, dropout=0.0):
    base = [Linear(8, 16, bias=False, dtype=torch.bfloat16) for _ in range(2)]
    return [lora.LoraLinear(m, 8, 16, dropout) for m in base] if adapters else base


@pytest.mark.parametrize("adapters", [False, True])
def test_taken_outside_autograd_only(fused, adapters):
    pair = _pair(adapters)
    assert fused(*pair) is None
    with torch.no_grad():
        assert fused(*pair) == "fused"


def test_adapters_that_do_not_ride_in_the_base_gemm_stay_as_they_are(fused):
    with torch.no_grad():
        assert fused(*_pair(True, dropout=0.1)) is None
        gate, up = _pair(True)
        up.base_layer.weight.requires_grad_(True)       # base, factors and sum are separate calls then, under autograd as well
        assert fused(gate, up) is None
        assert fused(_pair(True)[0], _pair(False)[0]) is None
        assert fused(*[nn.Linear(8, 16, bias=False, dtype=torch.bfloat16) for _ in range(2)]) is None


def _dual(f, x):
    with torch.autograd.forward_ad.dual_level():
        return f(x)


@pytest.mark.parametrize("around", [
    lambda f, x: torch.jit.trace(lambda t: (f(t), t)[1], x, check_trace=False),
    lambda f, x: torch.vmap(lambda t: (f(t), t)[1])(x[None]),
    lambda f, x: torch.func.jvp(lambda t: (f(t), t)[1], (x,), (x,)),
    _dual,
], ids=["trace", "vmap", "jvp", "dual level"])
def test_tracing_and_transforms_keep_the_autograd_functions(fused, around):
    seen, pair = [], _pair(False)
    with torch.no_grad():
        around(lambda t: seen.append((fused(*pair, t), ops.direct_calls())), torch.zeros(2, 8, dtype=torch.bfloat16))
        assert seen == [(None, False)] and ops.direct_calls()
    assert not ops.direct_calls()
