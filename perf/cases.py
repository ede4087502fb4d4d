"""The work that users of this package have it do, as cases to time.

Training steps of ``Trainer.step`` on rows as the packer lays them out, prompts and multi-step decoding through the runner
that ``build_runner`` gives (what the engine schedules), for the dense, sparse and hybrid families.  Models are the package's
own presets at full width, with the number of layers that a case names; weights, adapters, cached keys and token ids are
random.  A language-model head whose row ``next(t)`` points along the embedding of ``t`` makes the generating cases' next
token distributions as peaked as a trained model's, so that rounding does not change what is drawn.
"""
from __future__ import annotations

import dataclasses
import math
import random

import numpy as np
import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from art_b200.engine.factory import build_runner
from art_b200.engine.runner import SeqView
from art_b200.models.config import resolve_config
from art_b200.models.weights import LoraConfig, init_hybrid_weights, init_lora, linear_shapes, lora_key
from art_b200.trainer.trainer import TrainHyper, Trainer

DEV = "cuda"
BLOCK = 16                  # tokens of a cache block: the engine's default
EMBED_STD = 4.0             # the embedding stays the larger part of the residual stream
GREEDY_PEAK, SAMPLED_PEAK = 14.0, 18.0      # about the logit of the likeliest token: 0.9 and more of the mass
HYBRID_EMBED = 14.0
FEW = 200                   # of fewer numbers the error against 64 bits is a matter of chance
LORA = LoraConfig()         # rank 8, alpha 16


def listed():
    return [
        # one packed row is one optimizer step: what the service does unless told otherwise, on the smallest preset
        {"name": "train-small", "kind": "train", "model": "qwen2.5-0.5b", "layers": 24, "rows": 1, "seq": 2048, "prompt": 301, "completion": 333, "siblings": 4,
         "beta": 0.0, "micro": 8192},
        # the same on the model of the headline benchmark
        {"name": "train-row", "kind": "train", "model": "qwen2.5-7b", "layers": 8, "rows": 1, "seq": 2048, "prompt": 187, "completion": 289, "siblings": 6,
         "beta": 0.0, "micro": 8192},
        # a micro-batch of the headline benchmark: 8 rows of one prompt and its completions
        {"name": "train-batch", "kind": "train", "model": "qwen2.5-7b", "layers": 4, "rows": 8, "seq": 2048, "prompt": 512, "completion": 512, "siblings": 3,
         "beta": 0.0, "micro": 16384},
        # long multi-turn trajectories with a KL term against the base model
        {"name": "train-long-kl", "kind": "train", "model": "qwen3-8b", "layers": 2, "rows": 1, "seq": 16384, "prompt": 2041, "completion": 4703, "siblings": 3,
         "beta": 0.04, "micro": 16384},
        # a mixture of experts, adapters on every expert
        {"name": "train-experts", "kind": "train", "model": "qwen3-30b-a3b", "layers": 1, "rows": 4, "seq": 2048, "prompt": 405, "completion": 380, "siblings": 4,
         "beta": 0.0, "micro": 8192},
        # prompts of a rollout group as they arrive: ragged, over four resident adapters
        {"name": "prefill-batch", "kind": "prefill", "model": "qwen2.5-7b", "layers": 8, "seqs": 24, "new_lo": 130, "new_hi": 1100, "cached": 0, "adapters": 4,
         "temperature": 1.0},
        # the next turn of a conversation whose earlier turns are in the prefix cache
        {"name": "prefill-turn", "kind": "prefill", "model": "qwen3-8b", "layers": 8, "seqs": 1, "new_lo": 203, "new_hi": 203, "cached": 1504, "adapters": 1,
         "temperature": 0.0},
        # one user of the base model
        {"name": "decode-one", "kind": "decode", "model": "qwen2.5-3b", "layers": 36, "seqs": 1, "ctx_lo": 777, "ctx_hi": 777, "adapters": 0, "steps": 16,
         "temperature": 0.0},
        # agents with long contexts
        {"name": "decode-long", "kind": "decode", "model": "qwen3-8b", "layers": 8, "seqs": 48, "ctx_lo": 2000, "ctx_hi": 6000, "adapters": 1, "steps": 16,
         "temperature": 0.0},
        # the rollouts of the headline benchmark: 256 sequences over four adapters, prompts of 512 and up to 1536 new tokens
        {"name": "decode-batch", "kind": "decode", "model": "qwen2.5-7b", "layers": 8, "seqs": 256, "ctx_lo": 512, "ctx_hi": 2032, "adapters": 4, "steps": 16,
         "temperature": 1.0},
        # the hybrid family: linear attention of two kinds and latent attention
        {"name": "hybrid-prefill", "kind": "hybrid-prefill", "model": "nikelix-1b", "layers": 16, "seqs": 12, "new_lo": 170, "new_hi": 1300},
        {"name": "hybrid-decode", "kind": "hybrid-decode", "model": "nikelix-1b", "layers": 16, "seqs": 40, "ctx_lo": 120, "ctx_hi": 500, "steps": 16},
    ]


def draw(rng: random.Random):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["train", "train", "train", "prefill", "prefill", "decode", "decode", "decode", "hybrid-prefill", "hybrid-decode"])
    if kind == "train":
        model, layers, most = rng.choice([("qwen2.5-0.5b", 24, 8192), ("qwen2.5-7b", 4, 16384), ("qwen3-8b", 2, 16384), ("qwen3-30b-a3b", 1, 8192)])
        seq = 2048 * rng.choice([1, 1, 1, 2, 3, 4, 5, 8])       # the packer's row lengths are multiples of 2048
        seq = min(seq, most)
        rows = min(log(1, 8), max(1, most // seq))
        prompt = log(40, seq // 3)
        return {"kind": kind, "model": model, "layers": layers, "rows": rows, "seq": seq, "prompt": prompt, "completion": log(60, (seq - prompt) // 2),
                "siblings": rng.randint(1, 6), "beta": rng.choice([0.0, 0.0, 0.04]), "micro": rng.choice([8192, 16384])}
    if kind == "prefill":
        seqs = log(1, 24)
        lo = log(30, 1100)
        hi = min(lo * 2, 26000 // seqs)
        return {"kind": kind, "model": rng.choice(["qwen2.5-7b", "qwen3-8b"]), "layers": 8, "seqs": seqs, "new_lo": min(lo, hi), "new_hi": hi,
                "cached": rng.choice([0, 0, BLOCK * log(1, 90)]) if seqs <= 8 else 0, "adapters": rng.randint(0, 4), "temperature": rng.choice([0.0, 1.0])}
    if kind == "decode":
        model, layers, top = rng.choice([("qwen2.5-3b", 36, 8), ("qwen2.5-7b", 8, 256), ("qwen3-8b", 8, 96)])
        seqs = log(1, top)
        lo = log(60, 3000)
        hi = max(lo, min(2 * lo, 330000 // seqs))
        return {"kind": kind, "model": model, "layers": layers, "seqs": seqs, "ctx_lo": min(lo, hi), "ctx_hi": hi, "adapters": rng.randint(0, 4), "steps": 16,
                "temperature": rng.choice([0.0, 1.0])}
    seqs = log(1, 48)
    lo = log(50, 900)
    hi = max(lo, min(2 * lo, 16000 // seqs))
    lo = min(lo, hi)
    if kind == "hybrid-prefill":
        return {"kind": kind, "model": "nikelix-1b", "layers": 16, "seqs": seqs, "new_lo": lo, "new_hi": hi}
    return {"kind": kind, "model": "nikelix-1b", "layers": 16, "seqs": seqs, "ctx_lo": min(lo, 400), "ctx_hi": min(hi, 500), "steps": 16}


# ---------------------------------------------------------------------------------------------- inputs
def config(case):
    cfg = resolve_config(case["model"])
    if case["kind"].startswith("hybrid"):
        cfg.layers = cfg.layers[:case["layers"]]
        return cfg
    return dataclasses.replace(cfg, num_layers=case["layers"])


def after(t, vocab):
    """The token that the planted head finds likeliest behind ``t``."""
    return (t * 48271 + 11) % vocab


def lengths(case, lo, hi):
    """The sequence lengths of a batch: a matter of the case, not of the seed."""
    r = random.Random(repr(sorted((k, v) for k, v in case.items() if k != "name")))
    return [r.randint(case[lo], case[hi]) for _ in range(case["seqs"])]


def base_weights(cfg, seed, peak=None):
    """Random weights in Hugging Face names.  ``peak``: plant a next token with about that logit in the head; without, all
    tokens are nearly equally likely (training: the probability ratios then stay in the clipping range)."""
    g = torch.Generator(device=DEV).manual_seed(seed)

    def rnd(*shape, std=0.02):
        return torch.randn(*shape, generator=g, device=DEV, dtype=torch.bfloat16).mul_(std)

    d, V = cfg.hidden_size, cfg.vocab_size
    out_std = 0.02 / math.sqrt(2 * cfg.num_layers)
    w = {"model.embed_tokens.weight": rnd(V, d, std=EMBED_STD if peak else 1.0)}
    for i in range(cfg.num_layers):
        p = f"model.layers.{i}."
        for name, (o, n) in linear_shapes(cfg).items():
            w[p + name + ".weight"] = rnd(o, n, std=out_std if name.endswith(("o_proj", "down_proj")) else 0.02)
        if cfg.qkv_bias:
            for name, width in (("q_proj", cfg.q_size), ("k_proj", cfg.kv_size), ("v_proj", cfg.kv_size)):
                w[p + f"self_attn.{name}.bias"] = rnd(width)
        if cfg.qk_norm:
            for name in ("q_norm", "k_norm"):
                w[p + f"self_attn.{name}.weight"] = 1 + rnd(cfg.head_dim, std=0.1)
        if cfg.is_moe:
            w[p + "mlp.gate.weight"] = rnd(cfg.num_experts, d, std=0.05)
        for name in ("input_layernorm", "post_attention_layernorm"):
            w[p + name + ".weight"] = 1 + rnd(d, std=0.1)
    w["model.norm.weight"] = torch.ones(d, device=DEV, dtype=torch.bfloat16)
    if peak:
        head = torch.empty_like(w["model.embed_tokens.weight"])
        head[after(torch.arange(V, device=DEV), V)] = w["model.embed_tokens.weight"] * (peak / (0.95 * d * EMBED_STD))
        w["lm_head.weight"] = head
    else:
        w["lm_head.weight"] = rnd(V, d, std=0.03 / math.sqrt(d))
    return w


def hybrid_weights(cfg, seed):
    """Random weights; the embedding, which is the head as well, is large enough to make its own token the likeliest next."""
    w = init_hybrid_weights(cfg, seed=seed, dtype=torch.bfloat16, device=DEV)
    w["embed"] = w["embed"] * (HYBRID_EMBED / math.sqrt(cfg.hidden_size))
    return w


def adapter(cfg, seed):
    """LoRA factors in the middle of a training run: B is no longer zero."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    out = {}
    for k, v in init_lora(cfg, LORA, seed=seed % 1000).items():
        out[k] = torch.randn(v.shape, generator=g, device=DEV) * 0.02 if "lora_B" in k else v.to(DEV)
    return out


def spans(case):
    """The pieces of a packed row: (kind, start, length, position of the first token, prompt's number, own number)."""
    S, out, at, gid = case["seq"], [], 0, 0
    r = random.Random(case["seq"] * 31 + case["prompt"] * 7 + case["completion"])
    while at < S:
        P = case["prompt"]
        if out and S - at < P + 32:
            break                                                   # what is left of the row is padding
        n = min(P, S - at)
        prompt_id = gid
        out.append(("prompt", at, n, 0, prompt_id, prompt_id))
        gid += 1
        at += n
        for _ in range(case["siblings"]):
            n = case["completion"] if S % 2048 == 0 and case["completion"] * case["siblings"] + P == S else max(8, int(case["completion"] * r.uniform(0.6, 1.3)))
            n = min(n, S - at)
            if n < 8:
                break
            out.append(("completion", at, n, P, prompt_id, gid))
            gid += 1
            at += n
    return out


def packed_rows(case, cfg, seed):
    """Packed rows in pinned host memory, as the service hands them to the trainer."""
    R, S = case["rows"], case["seq"]
    rng = np.random.default_rng(seed)
    tok = rng.integers(0, cfg.vocab_size, (R, S))
    gid, pid, pos = np.full((R, S), -1), np.full((R, S), -1), np.zeros((R, S), dtype=np.int64)
    mask, adv, wts, lp = np.zeros((R, S), dtype=bool), np.zeros((R, S)), np.zeros((R, S)), np.full((R, S), np.nan)
    for r in range(R):
        ids = rng.integers(-2 ** 62, 2 ** 62, 4096)
        end = 0
        for kind, at, n, p0, prompt_id, own in spans(case):
            s = slice(at, at + n)
            gid[r, s], pid[r, s], pos[r, s] = ids[own], ids[prompt_id], np.arange(p0, p0 + n)
            end = at + n
            if kind == "completion":
                mask[r, s], adv[r, s], wts[r, s] = True, rng.normal(), 1.0 / n
                lp[r, s] = -math.log(cfg.vocab_size) + 0.02 * rng.normal(size=n)
        tok[r, end:] = 0
    wts[mask] /= wts[mask].mean()
    out = {"tokens": tok, "group_ids": gid, "parent_ids": pid, "input_pos": pos, "assistant_mask": mask, "logprobs": lp.astype(np.float32),
           "advantages": adv.astype(np.float32), "weights": wts.astype(np.float32)}
    return {k: torch.from_numpy(v) for k, v in out.items()}


def tables(counts, seed):
    """Block tables of sequences that grow to ``counts`` tokens: blocks in an order that a used pool hands out."""
    need = [(n + BLOCK - 1) // BLOCK for n in counts]
    order = np.random.default_rng(seed).permutation(sum(need)).tolist()
    out, at = [], 0
    for n in need:
        out.append(order[at:at + n])
        at += n
    return out, sum(need)


def slots(blocks, lo, hi):
    return [blocks[t // BLOCK] * BLOCK + t % BLOCK for t in range(lo, hi)]


def fill_cache(kv, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    for t in kv.k + kv.v:
        t.normal_(generator=g)


def generation(case, seed):
    """Sizes and token ids of a prompt or decode batch."""
    cfg = config(case)
    rng = np.random.default_rng(seed)
    if case["kind"].endswith("prefill"):
        new = lengths(case, "new_lo", "new_hi")
        cached = [case.get("cached", 0)] * len(new)
        counts, first = [c + n for c, n in zip(cached, new)], cached
        held = counts
    else:
        counts = lengths(case, "ctx_lo", "ctx_hi")
        first = [n - 1 for n in counts]
        held = [n + case["steps"] for n in counts]
    toks = [rng.integers(0, cfg.vocab_size, n).tolist() for n in counts]
    bt, n_blocks = tables(held, seed)
    n_ad = case.get("adapters", 0)
    ad = [i % n_ad if n_ad else -1 for i in range(len(counts))]
    return cfg, toks, first, bt, n_blocks, ad


def peak_of(case):
    return SAMPLED_PEAK if case["temperature"] > 0 else GREEDY_PEAK


def prepare(case, seed):
    kind = case["kind"]
    cfg = config(case)
    if kind == "train":
        trainer = Trainer(cfg, base_weights(cfg, seed), LORA, adapter(cfg, seed + 1), device=DEV)
        rows = {k: v.pin_memory() for k, v in packed_rows(case, cfg, seed + 2).items()}
        hyper = TrainHyper(learning_rate=5e-6, beta=case["beta"], rows_per_optimizer_step=case["rows"], tokens_per_microbatch=case["micro"])
        return {"case": case, "trainer": trainer, "rows": rows, "hyper": hyper}
    cfg, toks, first, bt, n_blocks, ad = generation(case, seed)
    if kind.startswith("hybrid"):
        runner, kv = build_runner(cfg, hybrid_weights(cfg, seed), num_blocks=n_blocks, block_size=BLOCK, num_slots=len(toks), device=DEV)
        seqs = [SeqView(toks[i], 0, bt[i], -1, 0.0, seed + i, 0, state_slot=i) for i in range(len(toks))]
        if kind == "hybrid-decode":
            # the prompts but their last token are in the cache and the recurrent state
            runner.prefill([dataclasses.replace(s, upto=len(s.tokens) - 1) for s in seqs])
            seqs = [dataclasses.replace(s, num_cached=len(s.tokens) - 1) for s in seqs]
    else:
        runner, kv = build_runner(cfg, base_weights(cfg, seed, peak_of(case)), num_blocks=n_blocks, block_size=BLOCK, device=DEV, lora_cfg=LORA,
                                  max_loras=max(1, case["adapters"]))
        fill_cache(kv, seed + 3)
        for a in range(case["adapters"]):
            runner.set_adapter(a, adapter(cfg, seed + 100 + a))
        seqs = [SeqView(toks[i], first[i], bt[i], ad[i], case["temperature"], seed + i, 0) for i in range(len(toks))]
    if kind.endswith("decode"):     # step by step
        where = [s for t in range(case["steps"]) for i in range(len(toks)) for s in slots(bt[i], first[i] + t, first[i] + t + 1)]
    else:
        where = [s for i in range(len(toks)) for s in slots(bt[i], first[i], len(toks[i]))]
    return {"case": case, "runner": runner, "kv": kv, "seqs": seqs, "where": torch.tensor(where, device=DEV)}


def run(state):
    case = state["case"]
    if case["kind"] == "train":
        m = state["trainer"].step(state["rows"], state["hyper"])
        flat = state["trainer"].flat
        return {"loss": m["loss"], "grad_norm": m["grad_norm"], "grads": flat.grads[:flat.numel], "params": flat.params[:flat.numel]}
    if case["kind"].endswith("prefill"):
        tokens, logprobs = state["runner"].prefill(state["seqs"])
    else:
        tokens, logprobs = state["runner"].decode(state["seqs"], case["steps"])
    out = {"tokens": torch.tensor(tokens), "logprobs": torch.tensor(logprobs)}
    kv, where = state["kv"], state["where"]
    if case["kind"].startswith("hybrid"):
        out["latent"] = torch.stack([L["latent"].flatten(0, 1)[where] for L in kv.layers if "latent" in L])
        out["states"] = [L[k] for L in kv.layers for k in ("state", "shift") if k in L]
        return out
    for name, cache in (("k", kv.k), ("v", kv.v)):      # the keys and values that the pass wrote
        rows = torch.stack([t.flatten(0, 1)[where] for t in cache])
        n = len(state["seqs"]) if case["kind"] == "decode" else rows.shape[1]
        out[name] = rows[:, :n]
        if case["kind"] == "decode":
            out[name + "_later"] = rows[:, n:]          # of the steps behind the first: they follow from the drawn tokens
    return out


# ---------------------------------------------------------------------------------------------- the least work
def attended(case):
    """Query-key pairs of one packed row."""
    n, prompts = 0, {}
    for kind, at, length, _, prompt_id, _ in spans(case):
        prompts.setdefault(prompt_id, length if kind == "prompt" else 0)
        n += length * (length + 1) // 2 + (length * prompts[prompt_id] if kind == "completion" else 0)
    return n


def work(case):
    cfg = config(case)
    if case["kind"].startswith("hybrid"):
        return hybrid_work(case, cfg)
    d, V, L = cfg.hidden_size, cfg.vocab_size, cfg.num_layers
    shapes = linear_shapes(cfg)
    held = sum(o * n for o, n in shapes.values())
    active = held
    if cfg.is_moe:
        expert = 3 * d * cfg.moe_intermediate_size
        active = held - (cfg.num_experts - cfg.num_experts_per_tok) * expert + cfg.num_experts * d
    lora = LORA.r * sum(o + n for o, n in shapes.values())
    if case["kind"] == "train":
        tokens = case["rows"] * case["seq"]
        scored = case["rows"] * sum(s[2] for s in spans(case) if s[0] == "completion")
        pairs = case["rows"] * attended(case) * cfg.q_size
        passes = 3 if case["beta"] > 0 else 2           # forward, gradient of the inputs; the base model's forward
        flops = L * (2 * passes * active * tokens + (4 * (passes - 1) + 8) * pairs) + (2 * passes) * V * d * scored
        nbytes = 2 * (L * held + V * d) + 2 * tokens * d + 8 * 4 * L * lora + 45 * tokens
        return {"bytes": nbytes, "flops": flops}
    _, toks, first, _, _, _ = generation(case, 0)
    n = len(toks)
    row = 2 * 2 * cfg.kv_size * L                       # one token's keys and values
    ad = 2 * L * lora * case["adapters"]
    if case["kind"] == "prefill":
        new = sum(len(t) - c for t, c in zip(toks, first))
        pairs = sum((len(t) * (len(t) + 1) - c * (c + 1)) // 2 for t, c in zip(toks, first))
        return {"bytes": 2 * (L * held + V * d) + ad + row * (new + sum(first)) + 2 * new * d,
                "flops": 2 * new * L * active + 4 * pairs * cfg.q_size * L + 2 * n * V * d}
    steps = case["steps"]
    keys = sum(len(t) for t in toks) * steps + n * steps * (steps - 1) // 2
    return {"bytes": steps * (2 * (L * held + V * d) + ad) + row * (keys + n * steps),
            "flops": steps * n * 2 * (L * active + V * d) + 4 * keys * cfg.q_size * L}


def hybrid_work(case, cfg):
    _, toks, first, _, _, _ = generation(case, 0)
    d, V = cfg.hidden_size, cfg.vocab_size
    n, decode = len(toks), case["kind"].endswith("decode")
    steps = case["steps"] if decode else 1
    new = n * steps if decode else sum(len(t) for t in toks)
    params = cfg.num_params() - V * d
    nbytes, flops = steps * 2 * (params + V * d), 2 * new * params + 2 * n * steps * V * d
    for s in cfg.layers:
        if s.type == "latent_attention":
            row = 2 * (s.kv_rank + s.rot_dim)
            seen = [min(t, s.window) for x in toks for t in (range(len(x), len(x) + steps) if decode else range(1, len(x) + 1))]
            flops += 2 * sum(seen) * s.heads * (s.dim + s.rot_dim + s.vdim)
            nbytes += row * (sum(seen) + new if decode else new)
        else:
            flops += 6 * new * s.heads * s.dim * s.vdim
            nbytes += 4 * n * steps * s.heads * s.dim * s.vdim * (2 if decode else 1)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """bf16 operands and activations through the layers: about what the outputs are off the 64-bit result, or four times that
    where it leaves room for it."""
    if case["kind"] == "train":
        return {"rel": 0.03}
    if case["kind"].startswith("hybrid"):
        return {"rel": 0.02, "differ": 0.01}
    return {"rel": 0.03, "differ": 0.01}


# ---------------------------------------------------------------------------------------------- 64-bit restatement
def rms(x, w, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * w


def rotate(x, pos, cfg):
    """x [T, heads, head_dim], halves rotated against each other."""
    half = cfg.head_dim // 2
    ang = pos.double().unsqueeze(-1) * cfg.rope_theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) / half)
    c, s = ang.cos().unsqueeze(-2), ang.sin().unsqueeze(-2)
    a, b = x[..., :half], x[..., half:]
    return torch.cat([a * c - b * s, b * c + a * s], -1)


class Plain:
    """The decoder in 64 bits.  ``lora``: a dict of factors per set of rows (``rows_of``: set of each row) or one dict."""

    def __init__(self, cfg, w):
        self.cfg, self.w = cfg, w

    def W(self, name):
        return self.w[name].double()

    def linear(self, x, layer, module, loras):
        p = f"model.layers.{layer}.{module}"
        y = x @ self.W(p + ".weight").t()
        if p + ".bias" in self.w:
            y = y + self.W(p + ".bias")
        for rows, lora in loras:
            a, b = lora[lora_key(layer, module, "A")].double(), lora[lora_key(layer, module, "B")].double()
            up = LORA.scale * ((x if rows is None else x[rows]) @ a.t()) @ b.t()
            y = y + up if rows is None else y.index_add(0, rows, up)
        return y

    def qkv(self, x, i, pos, loras):
        cfg, p = self.cfg, f"model.layers.{i}."
        h = rms(x, self.W(p + "input_layernorm.weight"), cfg.rms_norm_eps)
        q, k, v = (self.linear(h, i, f"self_attn.{n}_proj", loras).view(h.shape[0], -1, cfg.head_dim) for n in "qkv")
        if cfg.qk_norm:
            q = rms(q, self.W(p + "self_attn.q_norm.weight"), cfg.rms_norm_eps)
            k = rms(k, self.W(p + "self_attn.k_norm.weight"), cfg.rms_norm_eps)
        return rotate(q, pos, cfg), rotate(k, pos, cfg), v

    def mlp(self, x, i, loras):
        cfg, p = self.cfg, f"model.layers.{i}."
        h = rms(x, self.W(p + "post_attention_layernorm.weight"), cfg.rms_norm_eps)
        if not cfg.is_moe:
            act = F.silu(self.linear(h, i, "mlp.gate_proj", loras)) * self.linear(h, i, "mlp.up_proj", loras)
            return self.linear(act, i, "mlp.down_proj", loras)
        prob = (h @ self.W(p + "mlp.gate.weight").t()).softmax(-1)
        top, which = prob.topk(cfg.num_experts_per_tok, dim=-1)
        if cfg.norm_topk_prob:
            top = top / top.sum(-1, keepdim=True)
        out = torch.zeros_like(h)
        for e in range(cfg.num_experts):
            t, k = (which == e).nonzero(as_tuple=True)
            act = F.silu(self.linear(h[t], i, f"mlp.experts.{e}.gate_proj", loras)) * self.linear(h[t], i, f"mlp.experts.{e}.up_proj", loras)
            out = out.index_add(0, t, self.linear(act, i, f"mlp.experts.{e}.down_proj", loras) * top[t, k].unsqueeze(-1))
        return out

    def close(self, x, o, i, loras):
        x = x + self.linear(o, i, "self_attn.o_proj", loras)
        return x + self.mlp(x, i, loras)


def masked_attention(q, k, v, mask, scale):
    def head(q, k, v):
        return (q @ k.t() * scale).masked_fill(~mask, float("-inf")).softmax(-1) @ v

    rep = q.shape[1] // k.shape[1]
    one = [checkpoint(head, q[:, h], k[:, h // rep], v[:, h // rep], use_reentrant=False) for h in range(q.shape[1])]
    return torch.stack(one, 1).flatten(1)


def exact_train(case, seed):
    cfg = config(case)
    m = Plain(cfg, base_weights(cfg, seed))
    start = adapter(cfg, seed + 1)
    lora = {k: v.double().requires_grad_(True) for k, v in start.items()}
    rows = {k: v.to(DEV) for k, v in packed_rows(case, cfg, seed + 2).items()}
    R, S = rows["tokens"].shape
    head = m.W("lm_head.weight")

    def logprobs(h, t):
        def part(h, t):
            z = h @ head.t()
            return z.gather(1, t.unsqueeze(1)).squeeze(1) - torch.logsumexp(z, 1)

        return torch.cat([checkpoint(part, h[i:i + 512], t[i:i + 512], use_reentrant=False) for i in range(0, h.shape[0], 512)])

    for r in range(R):
        tok, gid, pid, pos = (rows[k][r] for k in ("tokens", "group_ids", "parent_ids", "input_pos"))
        mask = torch.ones(S, S, dtype=torch.bool, device=DEV).tril() & ((gid[:, None] == gid) | (pid[:, None] == gid))
        sel = rows["assistant_mask"][r, 1:].nonzero().squeeze(1)
        tgt = tok[1:][sel]

        def score(loras):
            x = m.w["model.embed_tokens.weight"][tok].double()
            for i in range(cfg.num_layers):
                def layer(x, i=i):
                    q, k, v = m.qkv(x, i, pos, loras)
                    return m.close(x, masked_attention(q, k, v, mask, cfg.head_dim ** -0.5), i, loras)

                x = checkpoint(layer, x.requires_grad_(torch.is_grad_enabled()), use_reentrant=False)
            return logprobs(rms(x, m.W("model.norm.weight"), cfg.rms_norm_eps)[sel], tgt)

        new = score([(None, lora)])
        old, adv = rows["logprobs"][r, 1:][sel].double(), rows["advantages"][r, 1:][sel].double()
        w = rows["weights"][r, 1:][sel].double() / (sel.numel() + 1e-6) / R
        ratio = (new - old).exp()
        loss = (-torch.min(ratio * adv, ratio.clamp(0.8, 1.2) * adv) * w).sum()
        if case["beta"] > 0:
            with torch.no_grad():
                ref = score([])
            loss = loss + case["beta"] * (((ref - new).exp() - (ref - new) - 1) * w).sum()
        loss.backward()
    names = list(lora)
    if cfg.is_moe:      # the factors of one kind lie side by side, expert after expert
        kinds = [f"mlp.experts.{{}}.{leaf}" for leaf in ("gate_proj", "up_proj", "down_proj")]
        names = [k for k in names if ".experts." not in k] + [lora_key(i, kind.format(e), ab) for i in range(cfg.num_layers) for kind in kinds for ab in "AB"
                                                              for e in range(cfg.num_experts)]
    grads = torch.cat([lora[k].grad.flatten() for k in names])
    params = torch.cat([start[k].double().flatten() for k in names])
    norm = grads.norm()
    g = grads * min(1.0, float(0.1 / (norm + 1e-6)))
    # the first step of AdamW: both moments are corrected to the gradient itself
    params = params * (1 - 5e-6 * 0.1) - 5e-6 * g / (g.abs() + 1e-8)
    # of single numbers it is chance how far a rounding sum is off: the loss and the norm are compared with each other only
    return {"loss": None, "grad_norm": None, "grads": grads, "params": params}


def exact_generation(case, seed):
    cfg, toks, first, bt, n_blocks, ad = generation(case, seed)
    m = Plain(cfg, base_weights(cfg, seed, peak_of(case)))
    loras = [adapter(cfg, seed + 100 + a) for a in range(case["adapters"])]
    shape = (n_blocks * BLOCK, cfg.num_kv_heads, cfg.head_dim)

    class Cache:
        k = [torch.empty(shape, dtype=torch.bfloat16, device=DEV) for _ in range(cfg.num_layers)]
        v = [torch.empty(shape, dtype=torch.bfloat16, device=DEV) for _ in range(cfg.num_layers)]

    fill_cache(Cache, seed + 3)
    scale, rep = cfg.head_dim ** -0.5, cfg.num_heads // cfg.num_kv_heads
    decode = case["kind"] == "decode"
    # one step of prompts, or `steps` steps of one token a sequence; `own`: this pass's keys and values by layer and step
    own = [[] for _ in range(cfg.num_layers)]
    cur = [t[c:] for t, c in zip(toks, first)]
    all_t, all_lp = [], []
    past = [torch.tensor(slots(bt[s], 0, first[s]), device=DEV, dtype=torch.long) for s in range(len(toks))]
    if decode:
        longest = max(first)
        at = torch.zeros(len(toks), longest, dtype=torch.long, device=DEV)
        seen = torch.zeros(len(toks), longest, dtype=torch.bool, device=DEV)
        for s, p in enumerate(past):
            at[s, :len(p)], seen[s, :len(p)] = p, True
    for step in range(case["steps"] if decode else 1):
        flat = torch.tensor([t for c in cur for t in c], device=DEV)
        pos = torch.cat([torch.arange(f + step, f + step + len(c), device=DEV) for f, c in zip(first, cur)])
        cuts = np.cumsum([0] + [len(c) for c in cur]).tolist()
        which = torch.tensor([a for a, c in zip(ad, cur) for _ in c], device=DEV)
        sets = [((which == a).nonzero().squeeze(1), l) for a, l in enumerate(loras)]
        x = m.w["model.embed_tokens.weight"][flat].double()
        for i in range(cfg.num_layers):
            q, k, v = m.qkv(x, i, pos, sets)
            own[i].append((k, v))
            o = torch.empty(x.shape[0], cfg.num_heads, cfg.head_dim, dtype=torch.float64, device=DEV)
            if decode:
                n, half = len(toks), max(1, len(toks) // 8)
                for a in range(0, n, half):
                    b = min(n, a + half)
                    ks = torch.cat([Cache.k[i][at[a:b]].double()] + [e[0][a:b, None] for e in own[i]], 1)
                    vs = torch.cat([Cache.v[i][at[a:b]].double()] + [e[1][a:b, None] for e in own[i]], 1)
                    ok = F.pad(seen[a:b], (0, step + 1), value=True)
                    qg = q[a:b].view(b - a, cfg.num_kv_heads, rep, cfg.head_dim)
                    z = torch.einsum("sgrd,stgd->sgrt", qg, ks).mul_(scale).masked_fill_(~ok[:, None, None], float("-inf")).softmax(-1)
                    o[a:b] = torch.einsum("sgrt,stgd->sgrd", z, vs).flatten(1, 2)
            else:
                for s in range(len(toks)):
                    c = slice(cuts[s], cuts[s + 1])
                    n, f = cuts[s + 1] - cuts[s], first[s]
                    ks, vs = (torch.cat([t[past[s]].double(), u[c]]).repeat_interleave(rep, 1) for t, u in ((Cache.k[i], k), (Cache.v[i], v)))
                    ok = torch.ones(n, n + f, dtype=torch.bool, device=DEV).tril(f)
                    z = torch.einsum("qhd,khd->hqk", q[c], ks).mul_(scale).masked_fill_(~ok, float("-inf")).softmax(-1)
                    o[c] = torch.einsum("hqk,khd->qhd", z, vs)
            x = m.close(x, o.flatten(1), i, sets)
        last = torch.tensor(cuts[1:], device=DEV) - 1
        z = rms(x[last], m.W("model.norm.weight"), cfg.rms_norm_eps) @ m.W("lm_head.weight").t()
        lp, t = z.log_softmax(-1).max(-1)
        all_t.append(t)
        all_lp.append(lp)
        cur = [[u] for u in t.tolist()]
    out = {"tokens": torch.stack(all_t).int(), "logprobs": torch.stack(all_lp)}
    if not decode:
        out = {k: v[0] for k, v in out.items()}
    for name, j in (("k", 0), ("v", 1)):
        out[name] = torch.stack([e[0][j] for e in own])
        if decode:
            out[name + "_later"] = torch.stack([torch.cat([s[j] for s in e[1:]]) for e in own])
    if out["logprobs"].numel() < FEW:
        out["logprobs"] = None
    if case["temperature"] > 0:     # the draw is the product's own, and what follows from it
        out.update({k: None for k in out if k not in ("k", "v")})
    return out


def exact_hybrid(case, seed):
    """Nikelix in 64 bits: the sequences side by side, padded behind their ends, the recurrences token by token."""
    cfg, toks, first, _, _, _ = generation(case, seed)
    w, eps = hybrid_weights(cfg, seed), cfg.norm_eps
    decode = case["kind"] == "hybrid-decode"
    # greedy decoding of this model repeats a token: its head is its embedding
    seqs = [t + [t[-1]] * (case["steps"] - 1) if decode else t for t in toks]
    B, T = len(seqs), max(len(t) for t in seqs)
    ids = torch.zeros(B, T, dtype=torch.long, device=DEV)
    for b, t in enumerate(seqs):
        ids[b, :len(t)] = torch.tensor(t, device=DEV)
    n = torch.tensor([len(t) for t in seqs], device=DEV)
    last = torch.arange(B, device=DEV), n - 1
    latents, states = [], []

    def W(name):
        return w[name].double()

    def norm(x, name=None):
        y = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)
        return y if name is None else y * W(name)

    def turn(x, base):          # neighbours rotated against each other
        m = x.shape[-1] // 2
        ang = torch.arange(T, device=DEV, dtype=torch.float64)[:, None] * base ** (-torch.arange(m, device=DEV, dtype=torch.float64) / m)
        c, s = ang.cos(), ang.sin()
        if x.dim() == 4:
            c, s = c[:, None], s[:, None]
        a, b = x[..., 0::2], x[..., 1::2]
        return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)

    def recur(decay, k, v, q, bonus=None):
        S = torch.zeros(B, k.shape[2], k.shape[3], v.shape[3], dtype=torch.float64, device=DEV)
        out = torch.empty_like(v)
        for t in range(T):
            kv = k[:, t, :, :, None] * v[:, t, :, None]
            new = torch.addcmul(kv, S, decay[:, t, :, :, None])
            out[:, t] = torch.einsum("bhkv,bhk->bhv", new if bonus is None else S + bonus[..., None] * kv, q[:, t])
            S = torch.where((t < n)[:, None, None, None], new, S)
        states.append(S.transpose(2, 3))
        return out

    def mixer(s, h, p):
        H = s.heads
        if s.type == "latent_attention":
            q = (h @ W(p + "q").t()).view(B, T, H, s.dim + s.rot_dim)
            low = h @ W(p + "dkv").t()
            c, kr = norm(low[..., :s.kv_rank], p + "dkv.norm"), turn(low[..., s.kv_rank:], s.rope_base)
            latents.append(torch.cat([c, kr], -1))
            qr = turn(q[..., s.dim:], s.rope_base)
            k, v = (c @ W(p + "uk").t()).view(B, T, H, s.dim), (c @ W(p + "uv").t()).view(B, T, H, s.vdim)
            i = torch.arange(T, device=DEV)
            ok = (i[:, None] >= i) & (i[:, None] - i < (s.window or T + 1))
            out = torch.empty(B, T, H, s.vdim, dtype=torch.float64, device=DEV)
            for b in range(B):
                z = torch.einsum("qhd,khd->hqk", q[b, ..., :s.dim], k[b]) + torch.einsum("qhd,kd->hqk", qr[b], kr[b])
                out[b] = torch.einsum("hqk,khd->qhd", z.mul_(s.scale).masked_fill_(~ok, float("-inf")).softmax(-1), v[b])
            return out.flatten(2) @ W(p + "o").t()
        if s.type == "hgrn2":
            q = F.silu(h @ W(p + "q").t()).view(B, T, H, s.dim)
            v = (h @ W(p + "v").t()).view(B, T, H, s.vdim)
            low = W(p + "lower")
            f = (low + (1 - low) * torch.sigmoid(h @ W(p + "f").t() + W(p + "f.b"))).view(B, T, H, s.dim)
            return norm(recur(f, 1 - f, v, q), p + "norm").flatten(2) @ W(p + "o").t()
        prev = F.pad(h, (0, 0, 1, 0))[:, :-1]
        shift = h[last]
        mix = {m: h + (prev - h) * W(p + "mu." + m) for m in "rkvgw"}
        r, k, v = ((mix[m] @ W(p + m).t()).view(B, T, H, s.dim) for m in "rkv")
        decay = (-(torch.tanh(mix["w"] @ W(p + "w1").t()) @ W(p + "w2").t() + W(p + "w0")).exp()).exp().view(B, T, H, s.dim)
        out = norm(recur(decay, k, v, r, W(p + "u"))).flatten(2) * W(p + "norm") * F.silu(mix["g"] @ W(p + "g").t())
        states.append(shift)
        return out @ W(p + "o").t()

    x = norm(w["embed"][ids].double(), "embed.norm")
    hist = [x]
    for i, s in enumerate(cfg.layers):
        p = f"l{i}."
        x = x + cfg.residual_mult * norm(mixer(s, norm(x, p + "norm1"), p + "mix."), p + "norm1b")
        z = norm(x, p + "norm2") @ W(p + "mlp.up").t()
        a, b, c, e = W(p + "mlp.act").tolist()
        y = a * norm(z) + b * norm(z ** 2) + c * norm(z ** 3) + e
        x = x + cfg.residual_mult * norm(y @ W(p + "mlp.down").t(), p + "norm2b")
        hist.append(x)
        x = sum(g * t for g, t in zip(W(p + "dwa").tolist(), hist))
    start = n - (case["steps"] if decode else 1)
    rows = start[None] + torch.arange(case["steps"] if decode else 1, device=DEV)[:, None]
    lp = (norm(x[torch.arange(B, device=DEV)[None], rows], "final.norm") @ W("embed").t()).log_softmax(-1)
    lp, t = lp.max(-1)
    if decode:
        if not torch.equal(t, ids[last].expand_as(t)):
            return None
        latent = [c[torch.arange(B, device=DEV)[None], rows].flatten(0, 1) for c in latents]
    else:
        t, lp = t[0], lp[0]
        latent = [torch.cat([c[b, :len(toks[b])] for b in range(B)]) for c in latents]
    return {"tokens": t.int(), "logprobs": lp if lp.numel() >= FEW else None, "latent": torch.stack(latent), "states": states}


def exact(case, seed):
    if case["kind"] == "train":
        return exact_train(case, seed)
    with torch.no_grad():
        if case["kind"].startswith("hybrid"):
            return exact_hybrid(case, seed)
        return exact_generation(case, seed)
