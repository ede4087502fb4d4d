"""Rotation of whole tokens, against fp64, over the numbers of tokens a CTA takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,heads,hd,inverse", [(1, 1, 16, False), (5, 40, 128, False), (593, 3, 64, True), (2049, 16, 64, False),
                                                (4801, 5, 128, True), (300, 2, 256, False), (40, 1, 544, False)])
def test_rope(M, heads, hd, inverse):
    from art_b200.ops import elementwise as ew

    g = torch.Generator(device=DEV).manual_seed(M)
    buf = torch.randn(M, 8 + (heads + 1) * hd, device=DEV, generator=g).bfloat16()
    pos = torch.randint(0, 2000, (M,), device=DEV, generator=g, dtype=torch.int32)
    was = buf.clone()
    ew.rope_(buf, pos, 8, heads, hd, 1e6, inverse=inverse)
    assert torch.equal(buf[:, :8], was[:, :8]) and torch.equal(buf[:, 8 + heads * hd:], was[:, 8 + heads * hd:])
    x = was[:, 8:8 + heads * hd].double().view(M, heads, hd)
    ang = pos.double()[:, None] * 1e6 ** (-2 * torch.arange(hd // 2, device=DEV, dtype=torch.float64) / hd)
    c, s = ang.cos()[:, None], ang.sin()[:, None] * (-1 if inverse else 1)
    a, b = x[..., :hd // 2], x[..., hd // 2:]
    want = torch.cat([a * c - b * s, b * c + a * s], -1)
    # one rounding to bf16; an angle of up to 2000 rad is off by up to 2000 * 2^-20 in fp32 (an exponent of up to 20 in exp2)
    err = (buf[:, 8:8 + heads * hd].double().view(M, heads, hd) - want).abs()
    assert (err <= 2 ** -8 * want.abs() + 2000 * 2 ** -20 * torch.cat([a.abs() + b.abs()] * 2, -1)).all()
