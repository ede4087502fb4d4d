"""Decode attention with the keys of all sequences in even shares over the chip, against fp64."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("lens,Hq,Hkv,hd,bs", [
    ([777], 16, 2, 128, 16),                                  # one context in many shares
    ([0, 1, 31, 32, 33, 127, 128, 129, 0], 8, 8, 128, 16),    # edges of a tile and of a CTA's four; empty contexts
    ([5000, 3, 0, 2111], 28, 4, 128, 16),                     # several heads of a context per share, many shares per head
    ([33] * 700, 14, 2, 64, 16),                              # more pairs than CTAs, several sequences per thread of the scan
    ([257, 64, 1], 32, 2, 32, 12),                            # 16 query heads per kv head, blocks that are no power of two
    ([1500] * 64, 8, 8, 64, 32),
])
def test_even_shares(lens, Hq, Hkv, hd, bs):
    from art_b200.ops import paged

    g = torch.Generator(device=DEV).manual_seed(len(lens) + hd)
    need = [(n + bs - 1) // bs for n in lens]
    nblk = sum(need) + 3
    kc, vc = (torch.randn(nblk, bs, Hkv, hd, generator=g, device=DEV).bfloat16() for _ in range(2))
    order = torch.randperm(nblk, generator=torch.Generator().manual_seed(1))
    bt = torch.zeros(len(lens), max(need) + 1, dtype=torch.int32)
    at = 0
    for i, n in enumerate(need):
        bt[i, :n] = order[at:at + n]
        at += n
    q = torch.randn(len(lens), (Hq + 2 * Hkv) * hd, generator=g, device=DEV).bfloat16()
    ctx, bt = torch.tensor(lens, dtype=torch.int32, device=DEV), bt.to(DEV)
    ws = paged.even_decode_workspace(len(lens), Hq, Hkv, hd, DEV)
    out = torch.full((len(lens), Hq * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    paged.paged_decode_even(q, kc, vc, bt, ctx, Hq, Hkv, hd, out, ws)
    again = torch.empty_like(out)
    paged.paged_decode_even(q, kc, vc, bt, ctx, Hq, Hkv, hd, again, ws)        # the counters are as the first call found them
    assert torch.equal(out, again)
    for i in list(range(len(lens)))[:: max(1, len(lens) // 16)]:
        n = lens[i]
        if n == 0:
            assert not out[i].any()
            continue
        rows = (bt[i, :need[i]].long()[:, None] * bs + torch.arange(bs, device=DEV)).reshape(-1)[:n]
        k = kc.flatten(0, 1)[rows].double().repeat_interleave(Hq // Hkv, 1)
        v = vc.flatten(0, 1)[rows].double().repeat_interleave(Hq // Hkv, 1)
        s = torch.einsum("hd,lhd->hl", q[i, :Hq * hd].double().view(Hq, hd), k) / math.sqrt(hd)
        p = s.softmax(-1)
        ref = torch.einsum("hl,lhd->hd", p, v)
        # each weight and the result are rounded to bf16, by at most 2^-8 of themselves; sums are fp32
        bound = 2 ** -8 * (torch.einsum("hl,lhd->hd", p, v.abs()) + ref.abs()) * 1.02 + 1e-5
        assert ((out[i].double().view(Hq, hd) - ref).abs() <= bound).all()
        assert (out[i].double().view(Hq, hd) - ref).norm() <= 4e-3 * ref.norm()
