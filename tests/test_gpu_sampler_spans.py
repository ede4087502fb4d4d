"""The fused sampler's vocabulary spans at the edges of their tiles."""
import pytest
import torch

from .test_gpu_model import DEV, _status_clean, bf  # noqa: F401

pytestmark = pytest.mark.gpu


# rows at and over one and two 128-row tiles, below and at the CTA-pair limit; vocabularies of less than a tile, whole tiles of
# each width and a column more, fewer tiles than CTAs
@pytest.mark.parametrize("M,V", [(1, 40), (8, 160 * 151), (128, 256 * 148 + 8), (129, 224 * 75), (300, 33000), (511, 1000), (512, 20008)])
def test_sampler_spans(M, V):
    from art_b200.ops import paged

    h, w = bf(M, 128, seed=1), bf(V, 128, scale=0.5, seed=2)
    logits = h.float() @ w.float().t()
    seeds = torch.arange(M, dtype=torch.int32, device=DEV)
    tok, lp = paged.sample(h, w, torch.zeros(M, device=DEV), seeds)
    want = torch.log_softmax(logits, -1)
    # the products' sums run in another order: 128 bf16 products, 2^-20 of their size each
    assert float((want.max(-1).values - want.gather(1, tok.long()[:, None])[:, 0]).max()) < 1e-3
    torch.testing.assert_close(lp, want.gather(1, tok.long()[:, None])[:, 0], rtol=0, atol=2e-3)
    # with noise: the same draw as the sampler on materialised logits
    it = torch.full((M,), 1 / 0.8, device=DEV)
    a, la = paged.sample(h, w, it, seeds)
    b, lb = paged.sample_restricted(h, w, it, seeds, torch.zeros(M, dtype=torch.int32, device=DEV), torch.ones(M, device=DEV))
    assert float((a != b).float().mean()) <= 2 / M + 0.005 * (M > 100)       # a tie within rounding may go either way
    torch.testing.assert_close(la[a == b], lb[a == b], rtol=0, atol=2e-3)
