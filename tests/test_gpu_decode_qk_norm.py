"""The finish of a decode step's q|k|v product with a norm of each head, against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,Hq,Hkv,hd", [(1, 32, 8, 128), (37, 3, 1, 64), (5, 14, 2, 32), (9, 5, 5, 16), (3, 7, 1, 256)])
def test_head_norm_in_qkv_finish(M, Hq, Hkv, hd):
    from art_b200.ops import paged

    g = torch.Generator(device=DEV).manual_seed(hd + M)
    qs, kvs, kpad, eps = Hq * hd, Hkv * hd, 64, 1e-6
    N = qs + 2 * kvs
    ws = torch.randn(M, N + kpad, device=DEV, generator=g)
    y = ws[:, :N].double()
    qn, kn = (1 + 0.1 * torch.randn(hd, device=DEV, generator=g)).bfloat16(), (1 + 0.1 * torch.randn(hd, device=DEV, generator=g)).bfloat16()
    pos = torch.randint(0, 300, (M,), device=DEV, generator=g, dtype=torch.int32)
    slot = torch.randperm(64, device=DEV, generator=g)[:M].to(torch.int32)
    kc, vc = torch.zeros(4, 16, Hkv, hd, device=DEV, dtype=torch.bfloat16), torch.zeros(4, 16, Hkv, hd, device=DEV, dtype=torch.bfloat16)
    q_out = torch.empty(M, qs, device=DEV, dtype=torch.bfloat16)
    paged.decode_finalize_qkv(ws, M, Hq, Hkv, hd, kpad, pos, 1e4, slot, kc, vc, q_out, q_norm=qn, k_norm=kn, eps=eps)

    def want(t, heads, w):
        t = t.reshape(M, heads, hd)
        t = t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + eps) * w.double()
        ang = pos.double()[:, None] * 1e4 ** (-2 * torch.arange(hd // 2, device=DEV, dtype=torch.float64) / hd)
        c, s = ang.cos()[:, None], ang.sin()[:, None]
        a, b = t[..., :hd // 2], t[..., hd // 2:]
        return torch.cat([a * c - b * s, b * c + a * s], -1).reshape(M, heads * hd)

    rows = slot.long()
    for got, ref in ((q_out, want(y[:, :qs], Hq, qn)), (kc.view(-1, kvs)[rows], want(y[:, qs:qs + kvs], Hkv, kn)),
                     (vc.view(-1, kvs)[rows], y[:, qs + kvs:])):
        # one rounding to bf16 (at most 2^-8 of the value); the angle of up to 300 rad is off by about 2^-15 in fp32
        assert ((got.double() - ref).abs() <= 2 ** -8 * ref.abs() + 3e-4 * ref.abs().amax()).all()
    assert not ws[:, :N].any()
