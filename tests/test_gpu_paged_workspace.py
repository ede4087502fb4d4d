"""One workspace of the even decode attention for batches of several sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("Hq,Hkv,hd", [(28, 4, 128), (16, 16, 64), (32, 2, 32)])
def test_smaller_batches_between(Hq, Hkv, hd):
    from art_b200.ops import paged

    g = torch.Generator(device=DEV).manual_seed(hd)
    n, bs, ctx = 96, 16, 1000
    per = (ctx + bs - 1) // bs
    kc, vc = (torch.randn(n * per, bs, Hkv, hd, generator=g, device=DEV).bfloat16() for _ in range(2))
    bt = torch.arange(n * per, dtype=torch.int32, device=DEV).view(n, per)
    q = torch.randn(n, Hq * hd, generator=g, device=DEV).bfloat16()
    lens = torch.full((n,), ctx, dtype=torch.int32, device=DEV)

    def run(k, ws):
        out = torch.full((k, Hq * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
        return paged.paged_decode_even(q[:k], kc, vc, bt[:k], lens[:k], Hq, Hkv, hd, out, ws)

    ws = paged.even_decode_workspace(n, Hq, Hkv, hd, DEV)
    for k in (n, 3, n, 1, 50, n):
        assert torch.equal(run(k, ws), run(k, paged.even_decode_workspace(k, Hq, Hkv, hd, DEV)))
