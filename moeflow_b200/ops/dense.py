"""Dense projections of a decode step on tcgen05 (``csrc/skinny_gemm.cu``): a weight matrix streamed past a few tokens.

The reference leaves these to the serving engine; here they carry the shared expert and the router logits of the decode
model (the projections around its attention are library GEMMs).
"""

from __future__ import annotations

import ctypes as C

import torch

from . import _lib
from .kernels import make_tile_tmap, sm_count


class DenseProjection:
    """``out[t] = x[t] . W^T`` for a bf16 ``W [rows, K]`` (rows a multiple of 128, K of 64), or, with ``gate_up``,
    ``silu(min(gate, limit)) * clamp(up, +-limit)`` for ``W`` holding the gate rows and then the up rows (each a
    multiple of 64).  fp32 sums; bf16 or fp32 output."""

    def __init__(self, w: torch.Tensor, gate_up: bool = False, limit: float | None = None, out_cols: int = 0,
                 status: torch.Tensor | None = None, wait_ns: int = 2_000_000_000):
        rows, k = w.shape
        block = 64 if gate_up else 128
        self.outputs = rows // 2 if gate_up else rows
        if k % 64 or self.outputs % block or w.dtype != torch.bfloat16:
            raise ValueError("bf16 weights with K a multiple of 64 and rows in whole blocks expected")
        self.w, self.k, self.gate_up = w.contiguous(), k, gate_up
        self._device = w.device
        self._width = min(out_cols, self.outputs) if out_cols > 0 else self.outputs  # columns that are stored
        self.status = status if status is not None else torch.zeros(1, dtype=torch.int64, device=w.device)
        self.n_sms = sm_count(w.device.index or 0)
        self._lib = _lib.lib()
        self._tmap = make_tile_tmap(self.w, block)
        self._args = _lib.SkinnyArgs(k_blocks=k // 64, row_blocks=self.outputs // block, up_row_offset=self.outputs if gate_up else 0,
                                     out_cols=out_cols, limit=float(limit) if limit is not None else 0.0,
                                     status=self.status.data_ptr(), wait_ns=wait_ns)

    def _check(self, name: str, t: torch.Tensor, rows: int, dtypes: tuple) -> None:
        """The kernel takes raw pointers: what it indexes has to be there."""
        if t.dtype not in dtypes or t.device != self._device:
            raise ValueError(f"{name} must be {' or '.join(str(d) for d in dtypes)} on the weights' device")
        if t.dim() != 2 or t.shape[0] < rows or t.shape[1] < self._width or (t.stride(1) != 1 and self._width > 1):
            raise ValueError(f"{name} must hold {rows} rows of {self._width} adjacent values")

    def __call__(self, x: torch.Tensor, out: torch.Tensor, residual: torch.Tensor | None = None,
                 residual2: torch.Tensor | None = None) -> torch.Tensor:
        """Writes ``out[: T]`` for ``x [T, K]``: bf16 rows at any 16-byte pitch are read in place, other types, layouts and
        devices are copied first.  ``residual`` (bf16 ``[T, rows]``), or the bf16 sum ``residual + residual2``, is added
        to the bf16 product."""
        t = x.shape[0]
        if x.dim() != 2 or x.shape[1] != self.k:
            raise ValueError("token rows do not fit this projection")
        self._check("out", out, t, (torch.bfloat16, torch.float32))
        if out.shape[0] > 1 and out.stride(0) < self._width:
            raise ValueError("the rows of out overlap")
        if residual2 is not None and residual is None:
            raise ValueError("residual2 is added to residual")
        for name, r in (("residual", residual), ("residual2", residual2)):
            if r is not None:
                self._check(name, r, t, (torch.bfloat16,))
        if residual is not None and out.dtype != torch.bfloat16:
            raise ValueError("a residual is added to a bf16 product")
        if t == 0:
            return out[:0]
        if x.device != self._device or x.dtype != torch.bfloat16:
            x = x.to(self._device, torch.bfloat16)
        if x.stride(1) != 1 or (t > 1 and (x.stride(0) < self.k or x.stride(0) % 8)) or x.data_ptr() % 16:
            x = x.clone(memory_format=torch.contiguous_format)
        a = self._args
        a.x, a.x_pitch, a.T = x.data_ptr(), (x.stride(0) if t > 1 else self.k) * 2, t
        a.out, a.out_pitch, a.out_fp32 = out.data_ptr(), out.stride(0), int(out.dtype == torch.float32)
        a.residual, a.residual_pitch = (residual.data_ptr(), residual.stride(0)) if residual is not None else (None, 0)
        a.residual2, a.residual2_pitch = (residual2.data_ptr(), residual2.stride(0)) if residual2 is not None else (None, 0)
        _lib.check(self._lib.mf_skinny_gemm(self._tmap, C.byref(a), int(self.gate_up), self.n_sms, _lib.stream_ptr()),
                   "dense projection")
        return out[:t]
