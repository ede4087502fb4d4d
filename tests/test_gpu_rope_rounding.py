"""The rotation bit for bit: one rounded product, then a fused multiply-add, in the same order for both of its forms."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def fma(a, b, c):
    # the product is exact in 64 bits; the sum's rounding there could only matter within 2^-29 of a tie
    return (a.double() * b.double() + c.double()).float()


@pytest.mark.parametrize("inverse", [False, True])
@pytest.mark.parametrize("M,heads,hd,theta", [(1, 1, 16, 1e4), (4801, 32, 128, 1e6), (2049, 16, 64, 1e4), (300, 2, 256, 1e6), (593, 3, 544, 1e6)])
def test_order_of_rounding(M, heads, hd, theta, inverse):
    from art_b200.ops import elementwise as ew

    g = torch.Generator(device=DEV).manual_seed(M + hd)
    x = torch.randn(M, heads * hd + 16, device=DEV, generator=g).bfloat16()
    pos = torch.randint(0, 8000, (M,), device=DEV, generator=g, dtype=torch.int32)
    half = hd // 2
    log2_theta = torch.tensor(math.log2(theta), dtype=torch.float32, device=DEV)
    inv_freq = torch.exp2(-log2_theta * (2.0 * torch.arange(half, device=DEV, dtype=torch.float32)) / hd)
    ang = pos.float()[:, None] * inv_freq
    c, s = ang.cos()[:, None], ang.sin()[:, None] * (-1 if inverse else 1)
    v = x[:, 8:-8].float().view(M, heads, hd)
    a, b = v[..., :half], v[..., half:]
    want = torch.cat([fma(a, c, -(b * s)), fma(b, c, a * s)], -1).bfloat16().flatten(1)
    for table in (None, inv_freq):
        y = x.clone()
        ew.rope_(y, pos, 8, heads, hd, theta, inverse=inverse, freqs=table)
        assert torch.equal(y[:, 8:-8], want)
