"""Fused LM-head log-prob + GRPO loss (``csrc/kernels/logprob_loss.cu``).

``forward`` returns per-token log-probs and accumulates the loss terms without ever
materialising logits; ``backward`` recomputes logit tiles, writes bf16 ``dlogits`` and
contracts them with the resident transposed LM head on the tcgen05 GEMM.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass

import torch

from . import _lib
from .gemm import gemm_tn

vp, ci, cf = ctypes.c_void_p, ctypes.c_int, ctypes.c_float
_bound: dict[str, object] = {}
_sigs = {
    "artb_logprob_parts": [ci, ci],
    "artb_logprob_partials": [vp, ci, vp, ci, vp, vp, vp, ci, ci, ci, ci, ci, ci, vp, vp],
    "artb_dlogits_inplace": [vp, ci, vp, vp, vp, ci, ci, ci, vp],
    "artb_grpo_tokens": [vp, ci, ci, vp, vp, vp, vp, cf, cf, cf, vp, vp, vp, vp, vp],
    "artb_logprob_dlogits": [vp, ci, vp, ci, vp, vp, vp, vp, ci, ci, ci, ci, ci, vp, vp],
}


def _f(name: str):
    fn = _bound.get(name)
    if fn is None:
        fn = getattr(_lib.kernels(), name)
        fn.argtypes = _sigs[name]
        fn.restype = ci
        _bound[name] = fn
    return fn


@dataclass
class LogprobResult:
    logprobs: torch.Tensor      # [M] fp32
    lse: torch.Tensor           # [M] fp32
    coef: torch.Tensor | None   # [M] dLoss/dlogprob (None for a stats-only pass)
    accum: torch.Tensor | None  # [4] fp32: sum(pg*w), sum(kl*w), #tokens with w != 0


def partials(hidden: torch.Tensor, lm_head: torch.Tensor, target: torch.Tensor, vocab_offset: int = 0,
             logits: torch.Tensor | None = None) -> tuple[torch.Tensor, int]:
    """Partial (max, sumexp, z_target) of one vocabulary shard: [parts, M, 4] fp32, and ``parts``.  ``logits`` ([M, ldl] fp32,
    ``ldl`` a multiple of 8) also receives the logits."""
    M, K = hidden.shape
    V = lm_head.shape[0]
    parts = _f("artb_logprob_parts")(M, V)
    part = torch.empty((parts, M, 4), dtype=torch.float32, device=hidden.device)
    rc = _f("artb_logprob_partials")(_lib.ptr(hidden), hidden.stride(0), _lib.ptr(lm_head), lm_head.stride(0),
                                     _lib.ptr(target), _lib.ptr(part), _lib.ptr(logits),
                                     logits.stride(0) if logits is not None else 0, M, V, K, parts, vocab_offset,
                                     _lib.ptr(_lib.status_word(hidden.device)), _lib.stream_ptr())
    _lib.check_rc(rc, "logprob_partials")
    return part, parts


def grpo_tokens(part: torch.Tensor, old_lp=None, adv=None, tok_w=None, ref_lp=None, eps_lo: float = 0.2,
                eps_hi: float = 0.2, beta: float = 0.0, accum: torch.Tensor | None = None) -> LogprobResult:
    splits, M, _ = part.shape
    dev = part.device
    lse = torch.empty(M, dtype=torch.float32, device=dev)
    lp = torch.empty(M, dtype=torch.float32, device=dev)
    coef = torch.empty(M, dtype=torch.float32, device=dev) if tok_w is not None else None
    if tok_w is not None and accum is None:
        accum = torch.zeros(4, dtype=torch.float32, device=dev)
    rc = _f("artb_grpo_tokens")(_lib.ptr(part), splits, M, _lib.ptr(old_lp), _lib.ptr(adv), _lib.ptr(tok_w),
                                _lib.ptr(ref_lp), eps_lo, eps_hi, beta, _lib.ptr(lse), _lib.ptr(lp), _lib.ptr(coef),
                                _lib.ptr(accum), _lib.stream_ptr())
    _lib.check_rc(rc, "grpo_tokens")
    return LogprobResult(lp, lse, coef, accum)


def forward(hidden, lm_head, target, old_lp=None, adv=None, tok_w=None, ref_lp=None, eps_lo=0.2, eps_hi=0.2,
            beta=0.0, accum=None) -> LogprobResult:
    """hidden [M,K] bf16, lm_head [V,K] bf16, target [M] int32 (next-token ids)."""
    part, _ = partials(hidden, lm_head, target)
    return grpo_tokens(part, old_lp, adv, tok_w, ref_lp, eps_lo, eps_hi, beta, accum)


def backward(hidden, lm_head, lm_head_t, target, lse, coef, dlogits_buf: torch.Tensor | None = None) -> torch.Tensor:
    """dH [M,K] bf16.  ``lm_head_t`` is the resident [K, ldo] transposed head (ldo = V padded to 8)."""
    M, K = hidden.shape
    V = lm_head.shape[0]
    ldo = lm_head_t.shape[1]
    if dlogits_buf is None or dlogits_buf.shape[0] < M:
        dlogits_buf = torch.empty((M, ldo), dtype=torch.bfloat16, device=hidden.device)
    dl = dlogits_buf[:M]
    rc = _f("artb_logprob_dlogits")(_lib.ptr(hidden), hidden.stride(0), _lib.ptr(lm_head), lm_head.stride(0),
                                    _lib.ptr(target), _lib.ptr(lse), _lib.ptr(coef), _lib.ptr(dl), ldo, M, V, K, 0,
                                    _lib.ptr(_lib.status_word(hidden.device)), _lib.stream_ptr())
    _lib.check_rc(rc, "logprob_dlogits")
    return gemm_tn(dl, lm_head_t)


LOGIT_ROWS = 2048     # at most this many rows' logits are alive at once, or half of the batch's (see forward_backward)


def kept_rows(M: int) -> int:
    """How many of ``M`` rows :func:`forward_backward` keeps the logits of at a time."""
    return min(M, max(LOGIT_ROWS, ((M + 1) // 2 + 255) // 256 * 256))


def forward_backward(hidden, lm_head, lm_head_t, target, old_lp, adv, tok_w, ref_lp=None, eps_lo=0.2, eps_hi=0.2, beta=0.0,
                     accum=None) -> tuple[LogprobResult, torch.Tensor]:
    """Loss terms of the rows of ``hidden`` and dLoss/dhidden [M,K] bf16, the logits computed once.

    The rows of a batch are independent, so it is cut into pieces whose fp32 logits are kept from the forward to the
    gradient: half of the rows, which is what all rows' bf16 dlogits would take, or ``LOGIT_ROWS`` where that is more.
    """
    M, K = hidden.shape
    V, ldl = lm_head.shape[0], lm_head_t.shape[1]
    piece = kept_rows(M)
    dh = torch.empty((M, K), dtype=torch.bfloat16, device=hidden.device)
    buf = torch.empty((piece, ldl), dtype=torch.float32, device=hidden.device)
    parts = []
    for m0 in range(0, M, piece):
        s = slice(m0, min(M, m0 + piece))
        n = s.stop - m0
        cut = lambda t: None if t is None else t[s]  # noqa: E731
        part, _ = partials(hidden[s], lm_head, target[s], logits=buf)
        res = grpo_tokens(part, cut(old_lp), cut(adv), cut(tok_w), cut(ref_lp), eps_lo, eps_hi, beta, accum)
        accum = res.accum
        rc = _f("artb_dlogits_inplace")(_lib.ptr(buf), ldl, _lib.ptr(target[s]), _lib.ptr(res.lse), _lib.ptr(res.coef), n, V, 0,
                                        _lib.stream_ptr())
        _lib.check_rc(rc, "dlogits_inplace")
        gemm_tn(buf.view(torch.bfloat16)[:n, :ldl], lm_head_t, out=dh[s])
        parts.append(res)
    if len(parts) == 1:
        return parts[0], dh
    join = lambda k: torch.cat([getattr(r, k) for r in parts])  # noqa: E731
    return LogprobResult(join("logprobs"), join("lse"), join("coef"), accum), dh


def reference_logprobs(hidden, lm_head, target):
    logits = hidden.float() @ lm_head.float().t()
    return logits.gather(-1, target.long().unsqueeze(-1)).squeeze(-1) - torch.logsumexp(logits, -1)
