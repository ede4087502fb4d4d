"""The table of a model's adapter factors: what it refuses."""
import pytest
import torch


def decoder(lcfg, lora=None):
    from art_b200.models.config import ModelConfig
    from art_b200.models.native import NativeDecoder
    from art_b200.models.weights import init_base_weights, init_lora

    cfg = ModelConfig(name="small", vocab_size=64, hidden_size=64, num_layers=2, num_heads=2, num_kv_heads=1, head_dim=32,
                      intermediate_size=96, qk_norm=False, qkv_bias=True)
    base = {k: v.to(torch.bfloat16) for k, v in init_base_weights(cfg, seed=0).items()}
    return NativeDecoder(cfg, base, lcfg, init_lora(cfg, lcfg) if lora is None else lora(cfg), device="cpu")


@pytest.mark.parametrize("r,targets", [(32, ("q_proj", "v_proj")), (64, ("v_proj",)), (64, ("up_proj",))])
def test_columns_behind_the_operands(r, targets):
    from art_b200.models.weights import LoraConfig

    with pytest.raises(ValueError, match="columns"):
        decoder(LoraConfig(r=r, target_modules=targets))


def test_factors_of_another_rank():
    from art_b200.models.weights import LoraConfig, init_lora

    with pytest.raises(ValueError, match="expected"):
        decoder(LoraConfig(r=16), lambda cfg: init_lora(cfg, LoraConfig(r=8)))
