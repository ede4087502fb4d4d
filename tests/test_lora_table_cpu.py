"""The table of a model's adapter factors: what it refuses, and models that are not on a GPU."""
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


def test_model_on_the_cpu():
    from art_b200.models.weights import LoraConfig

    m = decoder(LoraConfig())
    g = torch.Generator().manual_seed(1)
    m.flat.params.normal_(generator=g)
    m.refresh_lora()
    for lin in m.linears():
        lin.dA_acc.normal_(generator=g)
        lin.dB_acc.normal_(generator=g)
    m.export_grads()
    for lin in m.linears():
        for mem in lin.members:
            c = slice(mem.slot * lin.r, (mem.slot + 1) * lin.r)
            assert torch.equal(lin.A_cat[c], mem.a_view.bfloat16()) and torch.equal(lin.A_catT[:, c], lin.A_cat[c].t())
            assert torch.equal(lin.B_cat[mem.rows, c], (mem.b_view * lin.scale).bfloat16()) and torch.equal(lin.B_catT, lin.B_cat.t())
            assert torch.equal(mem.ga_view, lin.dA_acc[:, c].t()) and torch.equal(mem.gb_view, lin.dB_acc[mem.rows, c] * lin.scale)
    m.zero_grad()
    assert not any(t.any() for lin in m.linears() for t in (lin.dA_acc, lin.dB_acc))
