"""LoRA factor-gradient accumulation ``acc[C, 64] += p[M, C].T @ q[M, 64]``
(``csrc/kernels/lora_wgrad.cu``)."""
from __future__ import annotations

import ctypes

import torch

from . import _lib

_fn = None
_fn_pair = None


def accumulate_pair(acc1: torch.Tensor, p1: torch.Tensor, q1: torch.Tensor, acc2: torch.Tensor, p2: torch.Tensor, q2: torch.Tensor,
                    cols: int | None = None) -> None:
    """:func:`accumulate` for both factors of a projection, over the same rows, in one launch."""
    global _fn_pair
    if not p1.is_cuda or q1.shape[1] != 64:
        accumulate(acc1, p1, q1, cols=cols)
        accumulate(acc2, p2, q2, cols=cols)
        return
    if _fn_pair is None:
        _fn_pair = _lib.kernels().artb_lora_wgrad_pair
        vp, ci = ctypes.c_void_p, ctypes.c_int
        _fn_pair.argtypes = [vp, ci, vp, ci, vp, ci, ci] * 2 + [ci, ci, vp]
        _fn_pair.restype = ci
    for acc, p in ((acc1, p1), (acc2, p2)):
        assert acc.dtype == torch.float32 and acc.stride(1) == 1 and acc.shape[0] == p.shape[1] and p.shape[0] == p1.shape[0]
    _lib.check_rc(_fn_pair(_lib.ptr(p1), p1.stride(0), _lib.ptr(q1), q1.stride(0), _lib.ptr(acc1), acc1.stride(0), p1.shape[1],
                           _lib.ptr(p2), p2.stride(0), _lib.ptr(q2), q2.stride(0), _lib.ptr(acc2), acc2.stride(0), p2.shape[1],
                           p1.shape[0], cols or 64, _lib.stream_ptr()), "lora_wgrad_pair")


def accumulate(acc: torch.Tensor, p: torch.Tensor, q: torch.Tensor, transpose_out: bool = False,
               cols: int | None = None) -> None:
    """``acc`` fp32 [C, R]; ``p`` bf16 [M, C] (the wide operand); ``q`` bf16 [M, R], R == 64.

    ``cols``: columns of ``q`` from this one on are zero or not wanted, and those of ``acc`` unspecified (None: all count).

    ``transpose_out`` is accepted for call-site readability only: both LoRA gradients are
    stored with the wide dimension first, so the arithmetic is identical.
    """
    global _fn
    if not p.is_cuda:
        acc.add_(p.float().t() @ q.float())
        return
    M, C = p.shape
    R = q.shape[1]
    if R != 64:
        for c in range(0, R, 64):
            if cols is None or cols > c:
                accumulate(acc[:, c:c + 64], p, q[:, c:c + 64], cols=None if cols is None else min(64, cols - c))
        return
    if _fn is None:
        _fn = _lib.kernels().artb_lora_wgrad
        vp, ci = ctypes.c_void_p, ctypes.c_int
        _fn.argtypes = [vp, ci, vp, ci, vp, ci, ci, ci, ci, vp]
        _fn.restype = ci
    assert acc.dtype == torch.float32 and acc.stride(1) == 1 and acc.shape[0] == C
    _lib.check_rc(_fn(_lib.ptr(p), p.stride(0), _lib.ptr(q), q.stride(0), _lib.ptr(acc), acc.stride(0), M, C, cols or 64,
                      _lib.stream_ptr()), "lora_wgrad")
