"""Loss and gradient of the LM head from kept logits, against the two-pass form and a PyTorch oracle."""
import pytest
import torch

from .test_gpu_model import DEV, _status_clean, bf, rel_err  # noqa: F401

pytestmark = pytest.mark.gpu


# a padded row of 8 columns; one step of the in-place kernel and its neighbours; two pieces (one row in the second); pairs
@pytest.mark.parametrize("M,K,V", [(1, 64, 5), (130, 64, 4096), (37, 128, 4097), (260, 64, 8195), (2049, 64, 1000), (700, 192, 12289)])
def test_gradient_from_kept_logits(M, K, V):
    from art_b200.ops import logprob_loss as lpl

    h, w = bf(M, K, seed=1), bf(V, K, scale=0.2, seed=2)
    wt = torch.zeros(K, (V + 7) // 8 * 8, dtype=torch.bfloat16, device=DEV)
    wt[:, :V] = w.t()
    g = torch.Generator(device=DEV).manual_seed(3)
    tgt = torch.randint(0, V, (M,), device=DEV, dtype=torch.int32, generator=g)
    old = torch.full((M,), float("nan"), device=DEV)
    adv, tok_w = torch.randn(M, device=DEV, generator=g), torch.rand(M, device=DEV, generator=g)
    tok_w[::5] = 0
    res = lpl.forward(h, w, tgt, old, adv, tok_w)
    dh = lpl.backward(h, w, wt, tgt, res.lse, res.coef)
    accum = torch.zeros(4, device=DEV)
    kept, dk = lpl.forward_backward(h, w, wt, tgt, old, adv, tok_w, accum=accum)
    # the same products, the same arithmetic on the same fp32 logits
    torch.testing.assert_close(kept.logprobs, res.logprobs, rtol=1e-6, atol=1e-5)
    torch.testing.assert_close(accum[:3], res.accum[:3], rtol=1e-5, atol=1e-5)      # sums in another order
    assert rel_err(dk, dh) < 1e-3
    h32 = h.float().requires_grad_(True)
    lp = lpl.reference_logprobs(h32, w, tgt)
    (-(lp - lp.detach()).exp() * adv * tok_w).sum().backward()
    assert rel_err(dk, h32.grad) < 2e-2         # bf16 dlogits: 2^-9 each
