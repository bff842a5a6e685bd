"""The decoder's calls outside autograd on the GPU: what they give there is what the same calls give under autograd, tracing and transforms."""
import pytest
import torch

from nanorlhf_b200.models.qwen2 import Qwen2Config, Qwen2ForCausalLM

pytestmark = pytest.mark.gpu


def _mlp(width=256, ff=512):
    cfg = Qwen2Config(vocab_size=256, num_hidden_layers=1, hidden_size=width, intermediate_size=ff, num_attention_heads=2, num_key_value_heads=1,
                      head_dim=128)
    return Qwen2ForCausalLM.from_config(cfg, torch.bfloat16, "cuda", seed=0).model.layers[0].mlp


def test_a_traced_mlp_follows_its_inputs():
    mlp = _mlp()
    x, y = (torch.randn(300, 256, device="cuda").bfloat16() for _ in range(2))
    with torch.no_grad():
        traced = torch.jit.trace(mlp, x, check_trace=False)
        assert torch.allclose(traced(y).float(), mlp(y).float(), rtol=1e-2, atol=1e-2 * mlp(y).abs().max().item())      # one rounding apart at most


def test_forward_mode_is_refused_and_loses_no_tangent():
    mlp, fw = _mlp(), torch.autograd.forward_ad
    x = torch.randn(300, 256, device="cuda").bfloat16()
    with torch.no_grad(), fw.dual_level(), pytest.raises(NotImplementedError):
        mlp(fw.make_dual(x, x))
