"""Prompts of few rows through the finish kernels of a decode step, against the general path."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("hd,qk_norm", [(64, False), (128, True)])
@pytest.mark.parametrize("spans", [
    [(0, 1)],                                    # (cached, end) of every sequence
    [(0, 130)],
    [(144, 147)],                                # the new rows follow cached ones
    [(0, 7), (0, 33), (0, 250)],
    [(32, 50), (0, 65), (144, 400)],             # new rows in several places
    [(16, 512), (0, 16)],                        # 512 rows
])
def test_few_rows(hd, qk_norm, spans, monkeypatch):
    from art_b200.engine.kv_cache import KVCache
    from art_b200.engine.runner import NativeRunner, SeqView
    from art_b200.models.config import ModelConfig
    from art_b200.models.weights import LoraConfig, init_base_weights, init_lora

    cfg = ModelConfig(name="small", vocab_size=512, hidden_size=256, num_layers=2, num_heads=4, num_kv_heads=2, head_dim=hd,
                      intermediate_size=512, qk_norm=qk_norm, qkv_bias=not qk_norm)
    base = {k: v.to(torch.bfloat16) for k, v in init_base_weights(cfg, seed=0).items()}
    lcfg = LoraConfig()
    g = torch.Generator().manual_seed(5)
    lora = {k: torch.randn(v.shape, generator=g) * 0.05 if "lora_B" in k else v for k, v in init_lora(cfg, lcfg).items()}
    kv = KVCache(cfg.num_layers, 128, 16, cfg.num_kv_heads, hd, torch.device(DEV))
    runner = NativeRunner(cfg, lcfg, kv, base=base, max_loras=2, device=DEV)
    runner.set_adapter(1, {k: v.to(DEV) for k, v in lora.items()})
    order = torch.randperm(128, generator=g).tolist()
    seqs, at = [], 0
    for i, (nc, n) in enumerate(spans):
        need = (n + 15) // 16
        toks = torch.randint(0, cfg.vocab_size, (n,), generator=g).tolist()
        seqs.append(SeqView(toks, nc, order[at:at + need], 1 - 2 * (i % 2), 0.0, 0, 0))
        at += need
    want = [list(range(n - nc)) for nc, n in spans]
    held = [t.normal_(generator=torch.Generator(device=DEV).manual_seed(i)).clone() for i, t in enumerate(kv.k + kv.v)]

    def both(fused):
        monkeypatch.setenv("ARTB_DECODE_FUSED", fused)
        for t, h in zip(kv.k + kv.v, held):
            t.copy_(h)
        return runner.step_logits(seqs, want).double(), [t.clone() for t in kv.k + kv.v]

    a, ca = both("1")
    b, cb = both("0")
    # two layers of bf16 activations (2^-8 each) rounded in other places: a few roundings, of random sign, on every value
    assert (a - b).norm() < 4 * 2 ** -8 * b.norm()
    for x, y, h in zip(ca, cb, held):
        changed = (y != h).flatten(2).any(-1)
        assert torch.equal((x != h).flatten(2).any(-1), changed)          # the same slots were written
        assert (x.double() - y.double()).norm() < 4 * 2 ** -8 * y.double().norm()
