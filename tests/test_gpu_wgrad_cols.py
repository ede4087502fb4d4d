"""LoRA factor gradients over the used columns of the padded factors."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,C,cols", [(1, 8, 8), (31, 128, 16), (33, 136, 17), (64, 392, 24), (65, 896, 32), (1000, 3584, 33), (8200, 264, 64)])
def test_used_columns(M, C, cols):
    from art_b200.ops import wgrad

    g = torch.Generator(device=DEV).manual_seed(M + cols)
    p, q = (torch.randn(M, w, device=DEV, generator=g).bfloat16() for w in (C, 64))
    q[:, cols:] = 0
    acc = torch.ones(C, 64, device=DEV)
    wgrad.accumulate(acc, p, q, cols=cols)
    want = 1 + p.double().t() @ q.double()
    # products of bf16 are exact in fp32; M additions round by at most 2^-24 of the running sum each, random in sign
    assert ((acc.double() - want)[:, :cols].abs() <= 2 ** -24 * 8 * M ** 0.5 * (1 + p.double().abs().t() @ q.double().abs())[:, :cols]).all()


@pytest.mark.parametrize("M,C1,C2,cols", [(1, 8, 136, 8), (100, 896, 128, 24), (2048, 3584, 37888, 16), (513, 4864, 904, 40)])
def test_pair(M, C1, C2, cols):
    from art_b200.ops import wgrad

    g = torch.Generator(device=DEV).manual_seed(M)
    p1, p2, q1, q2 = (torch.randn(M, w, device=DEV, generator=g).bfloat16() for w in (C1, C2, 64, 64))
    a1, a2 = torch.zeros(C1, 64, device=DEV), torch.ones(C2, 64, device=DEV)
    wgrad.accumulate_pair(a1, p1, q1, a2, p2, q2, cols=cols)
    for acc, start, p, q in ((a1, 0, p1, q1), (a2, 1, p2, q2)):
        want, size = start + p.double().t() @ q.double(), start + p.double().abs().t() @ q.double().abs()
        assert ((acc.double() - want)[:, :cols].abs() <= 2 ** -24 * 8 * M ** 0.5 * size[:, :cols]).all()
