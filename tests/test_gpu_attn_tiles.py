"""Tensor-core attention over lists of key tiles: rows of many short groups, long rows, tiles of queries left out."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("lens,wanted", [
    ([128], None),
    ([1, 127, 129, 255, 300, 84], None),                 # groups that end inside, at and behind a tile's edge
    ([37] * 90 + [126], None),                           # several groups in every tile
    ([41472, 700, 1], None),                             # more tiles than threads of a CTA
    ([1504, 203, 85], [11, 12, 13]),                     # queries of three tiles only
])
def test_key_tile_lists(lens, wanted):
    from art_b200.ops import attention as A

    Hq, Hkv, hd = 3, 1, 128
    S = (sum(lens) + 127) // 128 * 128
    g = torch.Generator(device=DEV).manual_seed(S)
    gid = torch.cat([torch.full((n,), i) for i, n in enumerate(lens)] + [-1 - torch.arange(S - sum(lens))]).to(torch.int32).to(DEV)
    qkv = torch.randn(S, (Hq + 2 * Hkv) * hd, device=DEV, generator=g).bfloat16()
    plan = A.make_plan(gid, gid, S)
    tiles = wanted if wanted is not None else range(S // 128)
    if wanted is not None:
        plan.wanted = torch.zeros(S // 128, dtype=torch.uint8, device=DEV)
        plan.wanted[wanted] = 1
    out, _ = A.forward(qkv, Hq, Hkv, hd, plan, need_grad=False)
    rows = sorted({t * 128 + j for t in tiles for j in (0, 63, 127)})[-2000:]
    starts = torch.tensor([0] + lens).cumsum(0).tolist()
    for r in rows[:: max(1, len(rows) // 60)] + rows[-1:]:
        lo = next((a for a, n in zip(starts, lens) if a <= r < a + n), r)
        q = qkv[r, :Hq * hd].double().view(Hq, hd)
        k, v = qkv[lo:r + 1, Hq * hd:(Hq + 1) * hd].double(), qkv[lo:r + 1, (Hq + 1) * hd:].double()
        p = (q @ k.t() / math.sqrt(hd)).softmax(-1)
        ref = p @ v
        # each weight and the result are rounded to bf16, by at most 2^-8 of themselves; exponentials and sums are fp32
        bound = 2 ** -8 * (p @ v.abs() + ref.abs()) * 1.02 + 1e-5
        assert ((out[r].double().view(Hq, hd) - ref).abs() <= bound).all(), r
