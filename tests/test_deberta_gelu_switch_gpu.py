"""The reward model's intermediate layer with GELU in the GEMM's epilogue and, where the switch asks for it, as a pass of its own."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 130, 1000])
def test_the_switch_keeps_gemm_and_gelu_apart(rows, monkeypatch):
    from nanorlhf_b200.models.deberta_v3 import DebertaV3Config, _Intermediate
    layer = _Intermediate(DebertaV3Config(hidden_size=256, intermediate_size=512)).to("cuda", torch.bfloat16)
    x = torch.randn(rows, 256, device="cuda").bfloat16()
    with torch.no_grad():
        apart = torch.nn.functional.gelu(layer.dense(x))
        fused = layer(x)
        monkeypatch.setenv("NANORLHF_DEBERTA_GELU_FUSED", "0")
        assert torch.equal(layer(x), apart)
        want = torch.nn.functional.gelu(x.double() @ layer.dense.weight.double().T + layer.dense.bias.double())
    # one rounding against two of 2^-9 each
    assert (fused.double() - want).norm() < (apart.double() - want).norm() < 4e-3 * want.norm()
