"""Prompt rows that are not to be written to the cache, behind cached tokens or by themselves."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("spans", [[(32, 50)], [(0, 40), (48, 90)], [(16, 700), (0, 33)]])
def test_rows_not_written(hd, spans):
    from art_b200.engine.kv_cache import KVCache
    from art_b200.engine.runner import NativeRunner, SeqView
    from art_b200.models.config import ModelConfig
    from art_b200.models.weights import LoraConfig, init_base_weights

    cfg = ModelConfig(name="small", vocab_size=512, hidden_size=256, num_layers=2, num_heads=4, num_kv_heads=2, head_dim=hd,
                      intermediate_size=512, qk_norm=False, qkv_bias=True)
    base = {k: v.to(torch.bfloat16) for k, v in init_base_weights(cfg, seed=0).items()}
    kv = KVCache(cfg.num_layers, 128, 16, cfg.num_kv_heads, hd, torch.device(DEV))
    runner = NativeRunner(cfg, LoraConfig(), kv, base=base, max_loras=1, device=DEV)
    g = torch.Generator().manual_seed(2)
    order, at, seqs = torch.randperm(128, generator=g).tolist(), 0, []
    for nc, n in spans:
        blocks = order[at:at + (n + 15) // 16]
        at += len(blocks)
        toks = torch.randint(0, 512, (n,), generator=g).tolist()
        if nc:
            runner.prefill([SeqView(toks[:nc], 0, blocks, -1, 0.0, 0, 0)])
        seqs.append(SeqView(toks, nc, blocks, -1, 0.0, 0, 0))
    held = [t.clone() for t in kv.k + kv.v]
    got, _ = runner._prompt_forward(seqs, write_kv=False)
    assert all(torch.equal(t, h) for t, h in zip(kv.k + kv.v, held))
    want, _ = runner._prompt_forward(seqs, write_kv=True)
    # two layers of bf16 activations, rounded in other places where the rows are few
    assert (got.double() - want.double()).norm() < 4 * 2 ** -8 * want.double().norm()
    short = [SeqView(s.tokens, s.num_cached, s.blocks[:(s.num_cached + 15) // 16], -1, 0.0, 0, 0) for s in seqs]
    again, _ = runner._prompt_forward(short, write_kv=False)       # blocks for the cached tokens alone
    assert torch.equal(again, got)


@pytest.mark.parametrize("n,hd,copied", [(128, 128, False), (64, 64, False), (192, 64, False), (130, 128, True)])
def test_projection_is_the_buffer(n, hd, copied, monkeypatch):
    """Rows that fill whole tiles go to attention where the projection left them, LoRA columns beside them or not."""
    from art_b200.engine.kv_cache import KVCache
    from art_b200.engine.runner import NativeRunner, SeqView
    from art_b200.models.config import ModelConfig
    from art_b200.models.weights import LoraConfig, init_base_weights, init_lora
    from art_b200.ops import attention as attn_ops

    cfg = ModelConfig(name="small", vocab_size=512, hidden_size=256, num_layers=2, num_heads=4, num_kv_heads=2, head_dim=hd,
                      intermediate_size=512, qk_norm=False, qkv_bias=True)
    base = {k: v.to(torch.bfloat16) for k, v in init_base_weights(cfg, seed=0).items()}
    g = torch.Generator().manual_seed(n)
    lora = {k: torch.randn(v.shape, generator=g).to(DEV) * 0.05 if "lora_B" in k else v.to(DEV) for k, v in init_lora(cfg, LoraConfig()).items()}
    kv = KVCache(cfg.num_layers, 32, 16, cfg.num_kv_heads, hd, torch.device(DEV))
    runner = NativeRunner(cfg, LoraConfig(), kv, base=base, max_loras=1, device=DEV)
    runner.set_adapter(0, lora)
    toks = torch.randint(0, 512, (n,), generator=g).tolist()
    made, read = [], []
    qkv_of, attend = runner._qkv, attn_ops.forward

    def qkv(*a, **k):
        made.append(qkv_of(*a, **k))
        return made[-1]

    def forward(buf, *a, **k):
        read.append(buf)
        return attend(buf, *a, **k)

    monkeypatch.setattr(runner, "_qkv", qkv)
    monkeypatch.setattr(attn_ops, "forward", forward)
    for adapter in (-1, 0):
        made.clear(), read.clear()
        got, _ = runner._prompt_forward([SeqView(toks, 0, [], adapter, 0.0, 0, 0)], write_kv=False)
        assert [a.data_ptr() != b.data_ptr() for a, b in zip(made, read)] == [copied] * 2
        want, _ = runner._prompt_forward([SeqView(toks, 0, list(range(32)), adapter, 0.0, 0, 0)], write_kv=True)
        # two layers of bf16 activations, rounded in other places
        assert (got.double() - want.double()).norm() < 4 * 2 ** -8 * want.double().norm()
