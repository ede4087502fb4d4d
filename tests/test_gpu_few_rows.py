"""Products of few rows (stages that hold only as many rows of the first operand), against fp64."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M", [1, 8, 16, 17, 64, 65])
@pytest.mark.parametrize("N,K,K2", [(8, 8, 0), (136, 72, 64), (640, 2048, 0), (1312, 1096, 128)])
def test_few_rows(M, N, K, K2):
    from art_b200.ops.gemm import gemm_splitk_, gemm_tn

    g = torch.Generator(device=DEV).manual_seed(M * 7 + N)
    a, b = (torch.randn(r, K, device=DEV, generator=g).bfloat16() for r in (M, N))
    big = torch.full((256, K), float("nan"), device=DEV, dtype=torch.bfloat16)       # rows behind A that must not matter
    big[:M] = a
    a = big[:M]
    a2, b2 = (torch.randn(r, K2, device=DEV, generator=g).bfloat16() for r in (M, N)) if K2 else (None, None)
    want, size = a.double() @ b.double().t(), a.double().abs() @ b.double().abs().t()
    # exact products, fp32 sums: at most K roundings of 2^-24 of the running sum of sizes, seldom more than a few square roots
    bound = lambda s, k: 2 ** -24 * 8 * (k ** 0.5 + 8) * s + 1e-30
    for bn in (128, 160, 192, 224, 256):
        w2, s2 = (want + a2.double() @ b2.double().t(), size + a2.double().abs() @ b2.double().abs().t()) if K2 else (want, size)
        out = gemm_tn(a, b, a2=a2, b2=b2, out_dtype=torch.float32, bn=bn)
        assert ((out.double() - w2).abs() <= bound(s2, K + K2)).all(), bn
    for bn in (64, 128, 256):
        for splits in (1, 3):
            ws = torch.zeros(M, N, device=DEV)
            gemm_splitk_(ws, a, b, bn, splits)
            assert ((ws.double() - want).abs() <= bound(size, K)).all(), (bn, splits)


@pytest.mark.parametrize("M", [1, 16, 17, 64])
def test_few_rows_sampled(M):
    from art_b200.ops import paged

    g = torch.Generator(device=DEV).manual_seed(M)
    V, K = 152064, 256
    h, w = (torch.randn(r, K, device=DEV, generator=g).bfloat16() for r in (M, V))
    h = h * 0.2
    tok, lp = paged.sample(h, w, torch.zeros(M, device=DEV), torch.arange(M, device=DEV, dtype=torch.int32))
    logits = h.double() @ w.double().t()
    # greedy: the largest logit but for ties that fp32 sums decide
    best = logits.max(-1).values
    got = logits.gather(-1, tok.long().unsqueeze(-1)).squeeze(-1)
    assert ((best - got) <= 1e-4).all()
    assert ((lp.double() - torch.log_softmax(logits, -1).gather(-1, tok.long().unsqueeze(-1)).squeeze(-1)).abs() <= 2e-3).all()
