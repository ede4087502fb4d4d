"""Launches that overlap, weights requested early or not, against full stream order."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def whole(g, *shape):
    return torch.randint(-1, 2, shape, device=DEV, generator=g).bfloat16()


@pytest.mark.parametrize("M", [1, 16, 40, 128])
def test_chain_of_products(M):
    """Every launch reads what the one before it wrote.  Whole numbers: sums are exact in any order, so nothing may differ."""
    from art_b200.ops import paged
    from art_b200.ops.gemm import gemm_splitk_, gemm_tn, splitk_finalize

    g = torch.Generator(device=DEV).manual_seed(M)
    K, V, slots, cols = 1312, 8200, 2, 16
    w1, w2, b2 = whole(g, K, 64), whole(g, 640, K), whole(g, 19200, 64)
    w3, w4, wv = whole(g, 19200, 128), whole(g, 640 + 64, 19200), whole(g, V, 640)
    B = whole(g, 64, 640)
    adapter = torch.randint(-1, slots, (M,), device=DEV, generator=g, dtype=torch.int32)
    norm = whole(g, 640) + 2
    x0 = whole(g, M, 64)
    seeds, zero = torch.arange(M, device=DEV, dtype=torch.int32), torch.zeros(M, device=DEV)

    def chain(mode):
        ws2, ws4 = torch.zeros(M, 640, device=DEV), torch.zeros(M, 640 + 64, device=DEV)
        x, out = x0, []
        torch.cuda.synchronize()
        before = paged.set_pdl(mode)
        try:
            for _ in range(6):
                h1 = gemm_tn(x, w1, bn=128)                                 # one K block, fewer than the stages
                gemm_splitk_(ws2, h1, w2, 256, 8)                           # 21 K blocks in 8 slices of 3: the last is empty
                h2 = splitk_finalize(ws2, torch.empty(M, 640, device=DEV, dtype=torch.bfloat16))
                h3 = gemm_tn(h2[:, :128], w3, a2=h1[:, :64], b2=b2, bn=128)   # more tiles than CTAs, extra K within the stages
                gemm_splitk_(ws4, h3, w4, 128, 9)
                y, h4 = (torch.empty(M, 640, device=DEV, dtype=torch.bfloat16) for _ in range(2))
                paged.decode_finalize_norm(ws4, M, 640, 64, y, residual=h2, adapter=adapter, B_all=B, cols=cols, norm_w=norm, h_out=h4)
                tok, lp = paged.sample(h4, wv, zero, seeds)
                x = h4.sign()[:, :64].contiguous()
                out += [h1, h2, h3, y, h4, tok, ws2.clone(), ws4.clone()]
        finally:
            paged.set_pdl(before)
        return out

    want = chain(0)
    assert all(t.abs().max() > 0 for t in want[:5])
    for mode in (1, 2):
        for _ in range(3):
            for i, (a, b) in enumerate(zip(chain(mode), want)):
                assert torch.equal(a, b), (mode, i)


@pytest.mark.parametrize("n,adapters", [(5, True), (5, False), (40, True), (200, True), (200, False)])
def test_decode(n, adapters, monkeypatch):
    """Steps of a bucket of 8, of 64 and of 256 rows (products of one CTA, and of CTA pairs beside them)."""
    from art_b200.engine.kv_cache import KVCache
    from art_b200.engine.runner import NativeRunner, SeqView
    from art_b200.models.config import ModelConfig
    from art_b200.models.weights import LoraConfig, init_base_weights, init_lora

    cfg = ModelConfig(name="small", vocab_size=2048, hidden_size=512, num_layers=3, num_heads=4, num_kv_heads=2, head_dim=128,
                      intermediate_size=1024, qk_norm=False, qkv_bias=True)
    base = {k: v.to(torch.bfloat16) for k, v in init_base_weights(cfg, seed=0).items()}
    g = torch.Generator().manual_seed(5)
    # a token's embedding is most of its hidden row and the head points from it to the next token: draws are decided
    emb = torch.randn(cfg.vocab_size, cfg.hidden_size, generator=g)
    base["model.embed_tokens.weight"] = (emb * 4).bfloat16()
    base["lm_head.weight"] = (emb.roll(1, 0) * 20 / cfg.hidden_size).bfloat16()
    lcfg = LoraConfig()
    lora = {k: torch.randn(v.shape, generator=g) * 0.05 if "lora_B" in k else v for k, v in init_lora(cfg, lcfg).items()}
    kv = KVCache(cfg.num_layers, 1024, 16, cfg.num_kv_heads, cfg.head_dim, torch.device(DEV))
    order = torch.randperm(1024, generator=g).tolist()
    seqs = []
    for i in range(n):
        ctx = 10 + (i * 7) % 40
        toks = torch.randint(0, cfg.vocab_size, (ctx,), generator=g).tolist()
        seqs.append(SeqView(toks, ctx - 1, order[4 * i:4 * i + 4], i % 3 - 1 if adapters else -1, 0.0, 0, 0))
    held = [t.normal_(generator=torch.Generator(device=DEV).manual_seed(i)).clone() for i, t in enumerate(kv.k + kv.v)]
    got = {}
    for pdl in ("0", "1"):
        monkeypatch.setenv("ARTB_PDL", pdl)
        runner = NativeRunner(cfg, lcfg, kv, base=base, max_loras=2, device=DEV)
        for slot in range(2):
            runner.set_adapter(slot, {k: v.to(DEV) for k, v in lora.items()})
        for use in range(3):                     # eager, captured, replayed
            for t, h in zip(kv.k + kv.v, held):
                t.copy_(h)
            toks, lps = runner.decode(seqs, 6)
            got[pdl, use] = (torch.tensor(toks), torch.tensor(lps), torch.stack(kv.k + kv.v).double())
        runner.close()
    t0, l0, c0 = got["0", 0]
    assert torch.equal(t0[0], (torch.tensor([s.tokens[-1] for s in seqs]) + 1) % cfg.vocab_size)
    for t, lp, c in got.values():
        assert torch.equal(t, t0)
        # partial sums meet in any order: some activations are rounded to bf16 the other way
        assert (lp - l0).abs().max() < 0.05 and (c - c0).norm() < 2 ** -8 * c0.norm()


@pytest.mark.parametrize("n", [5, 40])
@pytest.mark.parametrize("which", ["aligned_design", "aligned_naselorn", "aligned_gaborax", "aligned_gaparax"])
def test_decode_of_hybrid_designs(which, n, monkeypatch):
    from art_b200.engine.factory import build_runner
    from art_b200.engine.runner import SeqView
    from art_b200.models.config import config_from_dict

    from . import hybrid_models
    from .hybrid_session import model, tokens

    d, w = model(getattr(hybrid_models, which)())
    runner, kv = build_runner(config_from_dict(d), w, num_blocks=8 * n, num_slots=n, dtype=torch.bfloat16)
    seqs = []
    for i in range(n):
        ctx = 20 + (i * 11) % 60
        seqs.append(SeqView(tokens(ctx, d["vocab"], 50 + i), 0, list(range(8 * i, 8 * i + 8)), -1, 0.0, 0, 0, state_slot=i, upto=ctx - 1))
    runner.prefill(seqs)
    for s in seqs:
        s.num_cached, s.upto = len(s.tokens) - 1, None
    tensors = [t for L in kv.layers for t in L.values() if torch.is_tensor(t)]
    held = [t.clone() for t in tensors]
    got = {}
    for pdl in ("0", "1"):
        monkeypatch.setenv("ARTB_PDL", pdl)
        runner.drop_graphs()
        for use in range(3):                     # eager, captured, replayed
            for t, h in zip(tensors, held):
                t.copy_(h)
            toks, lps = runner.decode(seqs, 6)
            got[pdl, use] = (torch.tensor(toks), torch.tensor(lps))
    t0, l0 = got["0", 0]
    for t, lp in got.values():
        # partial sums meet in any order and activations are bf16: draws agree until two tokens are as likely as one another
        same = (t == t0).int().cumprod(0).bool()
        upto = same.int().roll(1, 0)
        upto[0] = 1
        assert (lp - l0).abs()[upto.bool()].max() < 0.15
        assert same[0].float().mean() > 0.8
    runner.close()
