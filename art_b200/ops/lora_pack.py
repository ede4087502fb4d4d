"""Operand copies and gradient export of all LoRA factors of a model (``csrc/kernels/lora_pack.cu``)."""
from __future__ import annotations

import ctypes

import numpy as np
import torch

from . import _lib

TILE = 64
_ITEM = np.dtype([(k, np.uint64) for k in ("a", "b", "ga", "gb", "A_cat", "A_catT", "B_cat", "B_catT", "dA", "dB", "rows")]
                 + [(k, np.int32) for k in ("K", "n", "N", "kpad", "c0", "pad")])
_fn = None


def _f():
    global _fn
    if _fn is None:
        lib = _lib.kernels()
        if lib.artb_lora_item_bytes() != _ITEM.itemsize:
            raise _lib.NativeLibraryError("lora_pack: the library was built from other sources")
        _fn = lib.artb_lora_pack
        vp, ci = ctypes.c_void_p, ctypes.c_int
        _fn.argtypes, _fn.restype = [vp, vp, ci, ci, ctypes.c_float, ci, vp], ci
    return _fn


class LoraTable:
    """The members of ``linears`` (``models.native.LoraLinear``) as one table on the device.  Holds the linears, and with them
    every buffer that the table points to, and gives their gradient accumulators one allocation, cleared by one call.  Linears
    that are not on a GPU keep their own copies."""

    def __init__(self, linears: list):
        self.linears = [lin for lin in linears if lin.active]
        self.n_blocks = 0
        if not self.linears:
            return
        dev = self.linears[0].W.device
        self.r, self.scale = self.linears[0].r, self.linears[0].scale
        sizes = [t.numel() for lin in self.linears for t in (lin.dA_acc, lin.dB_acc)]
        self.acc = torch.zeros(sum(sizes), dtype=torch.float32, device=dev)
        parts = iter(self.acc.split(sizes))
        items, blocks = [], []
        for lin in self.linears:
            lin.dA_acc = next(parts).view(lin.dA_acc.shape)
            lin.dB_acc = next(parts).view(lin.dB_acc.shape)
            N, K = lin.W.shape
            for m in lin.members:
                tensors = (m.a_view, m.b_view, m.ga_view, m.gb_view, lin.A_cat, lin.A_catT, lin.B_cat, lin.B_catT, lin.dA_acc, lin.dB_acc, m.rows)
                assert all(t.is_contiguous() for t in tensors)
                n, r, c0 = m.rows.numel(), self.r, m.slot * self.r
                # the kernel takes these sizes on trust
                if c0 + r > lin.kpad:
                    raise ValueError(f"{m.module}: columns {c0} to {c0 + r} of low-rank operands with {lin.kpad}; adapt the modules "
                                     "before it as well, or use a lower rank")
                if lin.r != r or any(t.shape != (r, K) for t in (m.a_view, m.ga_view)) or any(t.shape != (n, r) for t in (m.b_view, m.gb_view)):
                    raise ValueError(f"{m.module}: factors {tuple(m.a_view.shape)} and {tuple(m.b_view.shape)}, ({r}, {K}) and ({n}, {r}) expected")
                tiles = (K + TILE - 1) // TILE + (n + TILE - 1) // TILE
                blocks += [(len(items), t) for t in range(tiles)]
                items.append(tuple(t.data_ptr() for t in tensors) + (K, n, N, lin.kpad, c0, 0))
        if dev.type != "cuda":
            return
        self.items = torch.from_numpy(np.array(items, dtype=_ITEM).view(np.uint8).copy()).to(dev)
        self.blocks = torch.from_numpy(np.array(blocks, dtype=np.int32)).to(dev)
        self.n_blocks = len(blocks)

    def _run(self, export: int) -> None:
        rc = _f()(_lib.ptr(self.items), _lib.ptr(self.blocks), self.n_blocks, self.r, self.scale, export, _lib.stream_ptr())
        _lib.check_rc(rc, "lora_pack")

    def refresh(self) -> None:
        if self.n_blocks:
            return self._run(0)
        for lin in self.linears:
            lin.refresh()

    def export_grads(self) -> None:
        if self.n_blocks:
            return self._run(1)
        for lin in self.linears:
            lin.export_grads()

    def zero_grad(self) -> None:
        if self.linears:
            self.acc.zero_()
