"""Backward of tree attention on tcgen05: head dim 64, and kv groups whose query heads are split over several CTAs."""
import pytest
import torch

from .test_gpu_model import _status_clean, bf, rel_err, tree_ids  # noqa: F401

pytestmark = pytest.mark.gpu


# one block; one head per group; seven heads over up to seven CTAs; a split that does not divide the group; many rows (two CTAs)
@pytest.mark.parametrize("rows,S,Hq,Hkv,hd,seg", [(1, 128, 3, 3, 64, 40), (1, 640, 7, 1, 64, 100), (2, 256, 10, 2, 64, 96), (1, 384, 5, 1, 128, 70),
                                                  (24, 256, 14, 2, 64, 256), (3, 256, 6, 2, 128, 128)])
def test_backward_with_split_groups(rows, S, Hq, Hkv, hd, seg):
    from art_b200.ops import attention as A

    M = rows * S
    qkv = bf(M, (Hq + 2 * Hkv) * hd, scale=0.7, seed=1)
    gid, pid = tree_ids(rows, S, seg)
    o, ctx = A.forward(qkv, Hq, Hkv, hd, A.make_plan(gid, pid, S, "native"))
    q32 = qkv.float().requires_grad_(True)
    ref = A.reference(q32, Hq, Hkv, hd, gid, pid, S)
    assert rel_err(o, ref) < 1e-2
    do = bf(M, Hq * hd, scale=0.5, seed=2)
    ref.backward(do.float())
    d = A.backward(do, ctx)
    for lo, hi in ((0, Hq), (Hq, Hq + Hkv), (Hq + Hkv, Hq + 2 * Hkv)):      # dQ, dK, dV each: bf16 operands and results
        assert rel_err(d[:, lo * hd:hi * hd], q32.grad[:, lo * hd:hi * hd]) < 2e-2
