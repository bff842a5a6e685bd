"""A projection whose sum with the residual could be formed in its GEMM: modules of other kinds are called as they are."""
import torch
import torch.nn as nn

from nanorlhf_b200 import ops
from nanorlhf_b200.models.lora import add_linear_forward
from nanorlhf_b200.models.qwen2 import Qwen2Config, Qwen2MLP


class Packed(nn.Module):
    """as quantised projections are: no weight, no bias"""

    def __init__(self, linear):
        super().__init__()
        self.inner = linear

    def forward(self, x):
        return self.inner(x)


def test_a_projection_without_a_bias_attribute(monkeypatch):
    monkeypatch.setattr(ops, "use_native", lambda t: True)             # the calls below are not made on the GPU: nothing is launched
    proj, x = Packed(nn.Linear(16, 8)), torch.randn(3, 16).bfloat16()
    with torch.no_grad():
        assert add_linear_forward(x, proj, torch.randn(3, 8).bfloat16()) is None


def test_an_mlp_with_such_a_projection_adds_the_residual():
    cfg = Qwen2Config.tiny()
    mlp = Qwen2MLP(cfg)
    x, h = torch.randn(3, cfg.hidden_size), torch.randn(3, cfg.hidden_size)
    with torch.no_grad():
        want = h + mlp(x)
        mlp.down_proj = Packed(mlp.down_proj)
        assert torch.equal(mlp(x, h), want)
