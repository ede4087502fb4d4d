"""Greedy draws among equal logits: the lowest token, wherever the tiles of the vocabulary begin and end."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


# rows that take tiles of each width (256, 224, 160 columns), one and several 128-row tiles, and CTA pairs
@pytest.mark.parametrize("M", [1, 16, 17, 64, 100, 129, 300, 512])
@pytest.mark.parametrize("V", [1000, 33000])
@pytest.mark.parametrize("twins", [(200, 261), (130, 262), (127, 128), (37, 995), (95, 161, 224), (3, 999)])
def test_lowest_token(M, V, twins):
    from art_b200.ops import paged

    g = torch.Generator(device=DEV).manual_seed(M)
    h = torch.rand(M, 64, device=DEV, generator=g).bfloat16() + 0.5
    w = torch.randn(V, 64, device=DEV, generator=g).bfloat16() * 0.01
    w[list(twins)] = torch.ones(64, device=DEV, dtype=torch.bfloat16)        # the largest logit by far, bit for bit the same
    zero, seeds = torch.zeros(M, device=DEV), torch.arange(M, device=DEV, dtype=torch.int32)
    tok, _ = paged.sample(h, w, zero, seeds)
    assert (tok == min(twins)).all()
    # shards of the vocabulary, merged in any order
    cut = (twins[0] // 8 + 1) * 8
    parts = [paged.sample_partials(h, w[:cut].contiguous(), zero, seeds), paged.sample_partials(h, w[cut:].contiguous(), zero, seeds, cut)]
    for order in (parts, parts[::-1]):
        assert (paged.sample_merge(torch.cat(order))[0] == min(twins)).all()
