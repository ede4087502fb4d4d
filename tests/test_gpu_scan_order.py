"""Portions of any lengths in one scan: taken by length, each gives what it gives alone."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("lens", [[5], [1, 40, 17], [3, 3, 3, 90, 0, 3], [1 + (37 * i) % 23 for i in range(256)], [1 + i % 5 for i in range(257)]])
def test_any_order_of_lengths(lens):
    from art_b200.ops import hybrid as hy

    H, dim, vdim = 2, 64, 64
    M = sum(lens)
    g = torch.Generator(device=DEV).manual_seed(M)
    q, v = (torch.randn(M, H * 64, device=DEV, generator=g).bfloat16() for _ in range(2))
    gate = torch.randn(M, H * dim, device=DEV, generator=g)
    bias, low = torch.randn(H * dim, device=DEV, generator=g), torch.rand(H * dim, device=DEV, generator=g) * 0.9

    def scan(rows, lengths):
        n = len(lengths)
        cu = torch.tensor([0] + lengths).cumsum(0).to(torch.int32).to(DEV)
        ctx, slot = torch.tensor(lengths, dtype=torch.int32, device=DEV), torch.arange(n, dtype=torch.int32, device=DEV)
        state = torch.full((n, H, vdim, dim), float("nan"), device=DEV)
        o = torch.empty(len(range(*rows.indices(M))), H * vdim, device=DEV)
        hy.linear_scan(hy.SCAN_HGRN2, hy.Out(q[rows], hy.KIND_BF16), None, hy.Out(v[rows], hy.KIND_BF16), hy.Out(gate[rows], hy.KIND_F32), bias, low, state,
                       cu, ctx, slot, n, H, dim, vdim, o)
        return o, state

    o, state = scan(slice(0, M), lens)
    at = 0
    for i, n in enumerate(lens):
        if n and (len(lens) < 20 or i % 29 == 0 or i == len(lens) - 1):
            # alone the portion may get column slices of another width: the same products, sums of eight parts in one order
            oi, si = scan(slice(at, at + n), [n])
            assert torch.allclose(o[at:at + n], oi, rtol=1e-5, atol=1e-5) and torch.allclose(state[i], si[0], rtol=1e-5, atol=1e-5)
        at += n
