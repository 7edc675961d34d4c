"""Python entry points of the standalone sm_100a kernels (router top-k, RMSNorm) and helpers shared by
the fused layer (tensor maps for the weight stream, SM count).  Each call launches on the current
CUDA stream, allocates only its outputs, and raises if the native library is missing.
"""

from __future__ import annotations

import ctypes as C
from functools import lru_cache

import torch

from ..config import MoEConfig
from . import _lib


def _need_cuda(t: torch.Tensor, what: str) -> None:
    if not t.is_cuda:
        raise ValueError(f"{what} must be a CUDA tensor")
    if not t.is_contiguous():
        raise ValueError(f"{what} must be contiguous")


@lru_cache(maxsize=8)
def sm_count(device_index: int) -> int:
    out = C.c_int()
    with torch.cuda.device(device_index):
        _lib.check(_lib.lib().mf_device_sm_count(C.byref(out)), "sm count")
    return out.value


def router_topk(
    logits: torch.Tensor,
    bias: torch.Tensor | None,
    cfg: MoEConfig,
    out_weights: torch.Tensor | None = None,
    out_ids: torch.Tensor | None = None,
) -> tuple[torch.Tensor, torch.Tensor]:
    """``logits [T, E]`` fp32 -> ``(weights [T, K] fp32, ids [T, K] int32)`` (see ``router.route``)."""
    _need_cuda(logits, "logits")
    if logits.dtype != torch.float32:
        raise ValueError("router_topk takes fp32 logits")
    n_tokens, n_experts = logits.shape
    if bias is not None:
        _need_cuda(bias, "bias")
        if bias.dtype != torch.float32 or bias.numel() != n_experts:
            raise ValueError("bias must be fp32 [E]")
    if cfg.scoring_func not in ("sigmoid", "softmax"):
        raise ValueError(f"unknown scoring function {cfg.scoring_func!r}")
    w = out_weights if out_weights is not None else torch.empty(n_tokens, cfg.top_k, dtype=torch.float32, device=logits.device)
    ids = out_ids if out_ids is not None else torch.empty(n_tokens, cfg.top_k, dtype=torch.int32, device=logits.device)
    _lib.check(
        _lib.lib().mf_router_topk(
            logits.data_ptr(), _lib.ptr(bias), w.data_ptr(), ids.data_ptr(), n_tokens, n_experts, cfg.top_k,
            cfg.n_group, cfg.topk_group, int(cfg.scoring_func == "sigmoid"), int(cfg.norm_topk_prob),
            float(cfg.routed_scaling_factor), _lib.stream_ptr(),
        ),
        "router_topk",
    )
    return w, ids


def rmsnorm(x: torch.Tensor, gamma: torch.Tensor, eps: float = 1e-6, out: torch.Tensor | None = None) -> torch.Tensor:
    """``out = x * rsqrt(mean(x^2) + eps) * gamma`` per row; bf16 in/out, fp32 math, one rounding."""
    _need_cuda(x, "x")
    _need_cuda(gamma, "gamma")
    if x.dtype != torch.bfloat16 or gamma.dtype != torch.bfloat16:
        raise ValueError("rmsnorm takes bf16 tensors")
    hidden = x.shape[-1]
    rows = x.numel() // hidden
    out = out if out is not None else torch.empty_like(x)
    _lib.check(
        _lib.lib().mf_rmsnorm(x.data_ptr(), gamma.data_ptr(), out.data_ptr(), rows, hidden, float(eps), _lib.stream_ptr()),
        "rmsnorm",
    )
    return out


def add_rmsnorm(x: torch.Tensor, add: torch.Tensor, gamma: torch.Tensor, eps: float = 1e-6) -> tuple[torch.Tensor, torch.Tensor]:
    """``(x + add, rmsnorm(x + add))`` in one launch; the sum is rounded to bf16 before it is normalised."""
    for name, t in (("x", x), ("add", add), ("gamma", gamma)):
        _need_cuda(t, name)
        if t.dtype != torch.bfloat16:
            raise ValueError("add_rmsnorm takes bf16 tensors")
    hidden = x.shape[-1]
    if add.shape != x.shape or gamma.numel() != hidden:
        raise ValueError("x, add and gamma do not fit each other")
    total, out = torch.empty_like(x), torch.empty_like(x)
    _lib.check(
        _lib.lib().mf_add_rmsnorm(x.data_ptr(), add.data_ptr(), gamma.data_ptr(), total.data_ptr(), out.data_ptr(),
                                  x.numel() // hidden, hidden, float(eps), _lib.stream_ptr()),
        "add_rmsnorm",
    )
    return total, out


def add_rmsnorm_logits(x: torch.Tensor, add: torch.Tensor, gamma: torch.Tensor, gate: torch.Tensor, experts: int, logits: torch.Tensor,
                       eps: float = 1e-6) -> tuple[torch.Tensor, torch.Tensor]:
    """``add_rmsnorm`` and the router logits of the normalised rows, ``logits[: rows] = h . gate[: experts]^T`` in fp32, in one
    launch."""
    for name, t in (("x", x), ("add", add), ("gamma", gamma), ("gate", gate)):
        _need_cuda(t, name)
        if t.dtype != torch.bfloat16:
            raise ValueError("add_rmsnorm_logits takes bf16 tensors")
    _need_cuda(logits, "logits")
    hidden = x.shape[-1]
    rows = x.numel() // hidden
    if add.shape != x.shape or gamma.numel() != hidden or gate.dim() != 2 or gate.shape[1] != hidden or gate.shape[0] < experts:
        raise ValueError("x, add, gamma and gate do not fit each other")
    if logits.dtype != torch.float32 or logits.dim() != 2 or logits.shape[0] < rows or logits.shape[1] != experts:
        raise ValueError("logits must be fp32 [rows, experts]")
    total, out = torch.empty_like(x), torch.empty_like(x)
    _lib.check(
        _lib.lib().mf_add_rmsnorm_logits(x.data_ptr(), add.data_ptr(), gamma.data_ptr(), total.data_ptr(), out.data_ptr(), rows, hidden,
                                         float(eps), gate.data_ptr(), experts, logits.data_ptr(), sm_count(x.device.index or 0),
                                         _lib.stream_ptr()),
        "add_rmsnorm_logits",
    )
    return total, out


def kv_append(k: torch.Tensor, v: torch.Tensor, k_cache: torch.Tensor, v_cache: torch.Tensor, pos: torch.Tensor) -> None:
    """Stores ``k`` / ``v`` (``[B, kv * d]``, equal row strides) as row ``pos`` (device int64 scalar) of the contiguous
    bf16 caches ``[B, kv, S, d]``."""
    B, kv, S, d = k_cache.shape
    for t in (k, v, k_cache, v_cache):
        if t.dtype != torch.bfloat16 or not t.is_cuda:
            raise ValueError("bf16 CUDA tensors expected")
    if (tuple(k.shape) != (B, kv * d) or v.shape != k.shape or v_cache.shape != k_cache.shape or k.stride(1) != 1 or v.stride() != k.stride()
            or not k_cache.is_contiguous() or not v_cache.is_contiguous()):
        raise ValueError("keys, values and caches do not fit each other")
    if pos.dtype != torch.int64 or pos.numel() != 1 or not pos.is_cuda:
        raise ValueError("pos must be a device int64 scalar")
    _lib.check(
        _lib.lib().mf_kv_append(k.data_ptr(), v.data_ptr(), k.stride(0), k_cache.data_ptr(), v_cache.data_ptr(), pos.data_ptr(),
                                B, kv, S, d, _lib.stream_ptr()),
        "kv append",
    )


def make_tile_tmap(x: torch.Tensor, box_rows: int) -> C.Array:
    """128-byte TMA descriptor over a contiguous ``x [rows, K]`` with boxes of ``box_rows`` rows x 128 bytes.

    Used for token operands whose rows are contiguous in expert-major order (boxes of up to 64 rows, as many as a tile holds;
    the e4m3 kernels take boxes of a whole tile) and for the weights of dense projections.  The buffer must outlive every
    launch that uses it.
    """
    _need_cuda(x, "token operand")
    if x.dim() != 2 or not x.is_contiguous():
        raise ValueError("the token operand must be a contiguous [rows, K] tensor")
    buf = (C.c_ubyte * 128)()
    _lib.check(_lib.lib().mf_make_tile_tmap(buf, x.data_ptr(), x.shape[0], x.shape[1], x.element_size(), box_rows),
               "tensor map")
    return buf


def make_weight_tmap(w: torch.Tensor) -> C.Array:
    """128-byte TMA descriptor over ``w`` viewed as ``[rows, K]`` (K innermost, 128 B x 128 row boxes)."""
    _need_cuda(w, "weight")
    k_elems = w.shape[-1]
    rows = w.numel() // k_elems
    buf = (C.c_ubyte * 128)()
    _lib.check(_lib.lib().mf_make_weight_tmap(buf, w.data_ptr(), rows, k_elems, w.element_size()), "tensor map")
    return buf
