"""GLM-5.3-Flash-shaped decoder built on the fused expert-parallel MoE layer.

Components (all inference-only, bf16, one process per GPU, attention TP=1 with data-parallel tokens,
DP = EP = world):

``SharedExpert``   the always-on SwiGLU MLP, on the tcgen05 kernel for dense projections of a decode step;
``MoEBlock``       RMSNorm (sm_100a kernel) -> router logits (``RouterLogits``: the same dense kernel, fp32 output) ->
                   routed experts (``FixedEPLayer``: fused route+dispatch, expert GEMMs, return push,
                   combine) + shared expert -> residual;
``Attention``      grouped-query attention over a static KV cache for single-token decode steps, with
                   PyTorch's scaled-dot-product attention (library code: attention is outside the scope of
                   the MoE backend and is served by the host engine in production);
``DecodeModel``    ``n_layers`` x (attention + MoE block), random-initialised, with one CUDA graph per
                   decode step.

In production the host engine (vLLM) owns model loading and attention and reaches the MoE layer
through ``moeflow_b200.integrations``; this module exists so that a whole decode step of the named
shape can be measured and tested without that engine.
"""

from __future__ import annotations

import math
from dataclasses import dataclass

import torch
import torch.nn.functional as F

from ..config import MoEConfig
from ..experts import swiglu_clamp
from ..fixed import FixedEPLayer


@dataclass(frozen=True)
class AttentionConfig:
    n_heads: int = 32
    n_kv_heads: int = 4
    head_dim: int = 128
    max_seq: int = 2304
    rope_theta: float = 10000.0


def _rmsnorm(x: torch.Tensor, gamma: torch.Tensor, eps: float) -> torch.Tensor:
    if x.is_cuda and x.dtype == torch.bfloat16:
        from ..ops.kernels import rmsnorm

        return rmsnorm(x, gamma, eps)
    xf = x.to(torch.float32)
    return (xf * torch.rsqrt(xf.pow(2).mean(-1, keepdim=True) + eps) * gamma.to(torch.float32)).to(x.dtype)


#: Up to this many router logits per step (sequences x experts) of rows of up to 4096 values come from the kernel that normalises the
#: rows, and of longer rows accordingly fewer: it reads the gate matrix once per sequence, the dense kernel once per 64.  Normalisation and
#: logits in a row of such pairs, cold gates, us, two launches / one: 36 experts, 1 sequence 6.5 / 4.2, 32 7.8 / 5.2, 64 8.7 / 9.2; 72
#: experts, 16 7.1 / 4.9, 32 7.8 / 7.9, 64 8.8 / 10.1; 288 experts, 4 7.3 / 6.1, 16 7.6 / 10.2.  Inside a decode step the second launch
#: costs more.  One layer of hidden 4096, 36 experts of 1536, e4m3: 4 sequences 150.3 / 144.6, 16 178.9 / 170.8, 40 208.8 / 203.9, 64 229.0 /
#: 222.5; bf16: 2 158.8 / 151.1, 64 319.2 / 312.3; 72 experts: 8 e4m3 204.2 / 197.0, 40 bf16 488.4 / 481.5, 64 508.1 / 507.6; but 1 sequence
#: 117.0 / 118.3, and 288 experts of 512, 16 sequences 234 to 240 / 241 to 246.  At hidden 8192, 36 experts of 1536: 24 sequences 489.8 / 488.4, 64
#: 509.2 / 513.5 (two layers' mean).
NORM_LOGITS = 2304
#: Below this hidden size a block with a shared expert keeps the two launches: its first half starts behind the normalisation, and the
#: dense kernel then runs beside it.  Hidden 2048, two layers' mean, two launches / one: intermediate 1536, 36 experts, 8 sequences 144.5 /
#: 147.1, 24 162.4 / 164.3, 40 174.5 / 177.6, 64 179.4 / 181.5; 1024, 72 experts, 32 183.3 / 189.4, 36 experts, 24 130.3 / 133.0; 512, 72
#: experts, 32 129.5 / 131.7 (8 sequences on 36 88.4 / 86.2); hidden 1024 within noise.  Without a shared expert (hidden 4096) one launch is
#: faster at all of these sizes: intermediate 512, 36 experts, 64 sequences 159.7 / 154.2; 1536, 72 experts, 32 428.1 / 421.3.
NORM_LOGITS_SHARED_HIDDEN = 4096


class SharedExpert:
    """Dense SwiGLU MLP ``w2 . swiglu(w13 . x)`` for up to ``capacity`` rows per call.  ``block_m`` is accepted for older
    call sites and selects nothing."""

    def __init__(self, w13: torch.Tensor, w2: torch.Tensor, capacity: int, limit: float | None, block_m: int = 64):
        self.w13, self.w2, self.C, self.limit = w13.contiguous(), w2.contiguous(), capacity, limit
        self.inter, self.hidden = w2.shape[-1], w2.shape[-2]
        self.cuda = w13.is_cuda and w13.dtype == torch.bfloat16 and self.hidden % 128 == 0 and self.inter % 128 == 0
        if not self.cuda:
            return
        from ..ops.dense import DenseProjection

        dev = w13.device
        self.act = torch.zeros(capacity, self.inter, dtype=torch.bfloat16, device=dev)
        self.out = torch.zeros(capacity, self.hidden, dtype=torch.bfloat16, device=dev)
        self.status = torch.zeros(1, dtype=torch.int64, device=dev)
        self._gate_up = DenseProjection(self.w13, gate_up=True, limit=limit, status=self.status)
        self._down = DenseProjection(self.w2, status=self.status)

    def begin(self, x: torch.Tensor, branch: torch.cuda.Stream, whole: bool = False) -> torch.Tensor | None:
        """The gate/up half of ``add_to(x, ..., begun=branch)`` on a branch of the graph that is being captured: next to the
        router, the dispatch and the start of the routed experts, which leave most SMs idle, instead of behind the routed
        experts (12 us of a decode layer).  ``whole``: the down half as well; returns the rows (valid behind the branch)."""
        branch.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(branch):
            self._gate_up(x, self.act)
            return self._down(self.act[: x.shape[0]], self.out) if whole else None

    def __call__(self, x: torch.Tensor) -> torch.Tensor:
        if not self.cuda:
            h = swiglu_clamp(x @ self.w13.transpose(0, 1), self.limit)
            return h @ self.w2.transpose(0, 1)
        return self._down(self._gate_up(x, self.act), self.out)

    def add_to(self, x: torch.Tensor, first: torch.Tensor, second: torch.Tensor, out: torch.Tensor,
               begun: torch.cuda.Stream | None = None) -> torch.Tensor:
        """``out = (first + second) + self(x)``, rounded to bf16 after every addition; the down projection adds (two
        element-wise launches less per layer).  ``begun``: ``begin(x, begun)`` has launched the first half.  cuda path
        only."""
        if begun is not None:
            torch.cuda.current_stream().wait_stream(begun)
            return self._down(self.act[: x.shape[0]], out, first, second)
        return self._down(self._gate_up(x, self.act), out, first, second)


class RouterLogits:
    """Router logits ``h . gate_w^T`` as fp32 ``[T, E]`` on the dense projection kernel (tcgen05, bf16 operands, fp32
    accumulation and fp32 output): the gate matrix's rows are padded to a multiple of 128 and only the E real columns
    are stored.  With it the MoE block issues no library GEMM.  ``block_m`` as in ``SharedExpert``."""

    def __init__(self, gate_w: torch.Tensor, capacity: int, block_m: int = 64):
        from ..ops.dense import DenseProjection

        E, H = gate_w.shape
        dev = gate_w.device
        if H % 64:
            raise ValueError("hidden size must be a multiple of 64")
        self.E, self.H, self.C = E, H, capacity
        self.w = torch.zeros((E + 127) // 128 * 128, H, dtype=torch.bfloat16, device=dev)
        self.w[:E] = gate_w.to(torch.bfloat16)
        self.logits = torch.zeros(capacity, E, dtype=torch.float32, device=dev)
        self.status = torch.zeros(1, dtype=torch.int64, device=dev)
        self._project = DenseProjection(self.w, out_cols=E, status=self.status)

    def __call__(self, h: torch.Tensor) -> torch.Tensor:
        return self._project(h, self.logits)

    def fits_norm(self, rows: int, shared: bool = False) -> bool:
        """Is ``after_norm`` the faster form?  ``shared``: in a block with a shared expert."""
        if not 0 < rows <= self.C or self.H > 16384 or (shared and self.H < NORM_LOGITS_SHARED_HIDDEN):
            return False
        return rows * self.E * max(self.H, 4096) <= NORM_LOGITS * 4096

    def after_norm(self, x: torch.Tensor, add: torch.Tensor, gamma: torch.Tensor, eps: float) -> tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
        """``(x + add, h = rmsnorm(x + add), router logits of h)`` in one launch."""
        from ..ops.kernels import add_rmsnorm_logits

        total, h = add_rmsnorm_logits(x, add, gamma, self.w, self.E, self.logits, eps)
        return total, h, self.logits[: x.shape[0]]


class MoEBlock:
    """Pre-norm MoE block: ``x + routed(norm(x)) + shared(norm(x))``."""

    def __init__(self, cfg: MoEConfig, routed: FixedEPLayer, gate_w: torch.Tensor, bias: torch.Tensor | None,
                 norm_w: torch.Tensor, shared: SharedExpert | None, eps: float = 1e-6, router: RouterLogits | None = None,
                 branch: torch.cuda.Stream | None = None):
        """``branch``: a stream that captured calls may put the shared expert's first half on."""
        self.cfg, self.routed, self.gate_w, self.bias, self.norm_w, self.shared, self.eps = cfg, routed, gate_w, bias, norm_w, shared, eps
        self.router, self.branch = router, branch

    def __call__(self, x: torch.Tensor, num_valid: torch.Tensor | None = None, add: torch.Tensor | None = None,
                 out: torch.Tensor | None = None) -> torch.Tensor:
        """``add``: summand of ``x`` that is still missing (the attention output).  ``out`` (contiguous bf16 ``[T, H]``,
        not ``x``) receives the result."""
        logits = None
        if add is not None and x.is_cuda and x.dtype == torch.bfloat16:
            from ..ops.kernels import add_rmsnorm

            if self.router is not None and x.dim() == 2 and self.router.fits_norm(x.shape[0], self.shared is not None):
                x, h, logits = self.router.after_norm(x, add, self.norm_w, self.eps)
            else:
                x, h = add_rmsnorm(x, add, self.norm_w, self.eps)
        else:
            x = x if add is None else x + add
            h = _rmsnorm(x, self.norm_w, self.eps)
        fused = self.shared is not None and self.shared.cuda and x.dtype == torch.bfloat16
        # only in a graph, where a branch costs the host nothing per step
        capturing = fused and self.branch is not None and self.routed.backend == "cuda" and torch.cuda.is_current_stream_capturing()
        begun = self.branch if capturing else None
        # one rank: the whole shared expert runs on the branch, and the routed experts' last kernel adds the three up, in rows of 16-byte
        # chunks; any other `out` is left to the shared expert's down projection
        wide = lambda t: t.shape == h.shape and t.dtype == h.dtype and t.device == h.device and t.is_contiguous() and t.data_ptr() % 16 == 0
        added = begun is not None and self.routed.adds_to_output and wide(x) and (out is None or wide(out))
        if begun is not None:
            beside = self.shared.begin(h, begun, whole=added)
        if logits is not None:
            pass
        elif self.router is not None:
            logits = self.router(h)
        else:
            logits = torch.matmul(h.to(self.gate_w.dtype), self.gate_w.transpose(0, 1)).to(torch.float32)
        if added:
            join = lambda: torch.cuda.current_stream().wait_stream(begun)
            return self.routed.forward_add(h, logits, self.bias, num_valid, x, beside, torch.empty_like(h) if out is None else out, join)
        routed = self.routed.forward(h, logits, self.bias, num_valid)[: x.shape[0]]
        if begun is not None or (fused and routed.dtype == torch.bfloat16):
            return self.shared.add_to(h, x, routed, torch.empty_like(h) if out is None else out, begun)
        y = x + routed
        if self.shared is not None:
            y = y + self.shared(h)
        return y if out is None else out.copy_(y)


class Attention:
    """Single-token GQA decode step over a static KV cache ``[B, n_kv, max_seq, d]`` (library SDPA and projections).

    The library's projections at these sizes, one after the other in a graph, cold weights, library / dense projection kernel, us:
    output (4096 x 4096) 1 sequence 13.7 / 10.2, 4 12.5 / 10.4, 16 10.8 / 10.9, 64 10.9 / 13.3; queries, keys and values (5120 x 4096)
    11.6 / 16.2, 12.0 / 16.4, 13.1 / 17.1, 12.1 / 22.9.  The dense kernel keeps a tensor map of its weights, though, and these may be
    exchanged, or changed through a view, between uncaptured steps."""

    def __init__(self, hidden: int, acfg: AttentionConfig, batch: int, device, seed: int):
        self.acfg, self.hidden, self.batch = acfg, hidden, batch
        g = torch.Generator(device=device).manual_seed(seed)
        q_out, kv_out = acfg.n_heads * acfg.head_dim, acfg.n_kv_heads * acfg.head_dim

        def w(rows, cols):
            return (torch.randn(rows, cols, generator=g, device=device) / math.sqrt(cols)).to(torch.bfloat16)

        self.wqkv, self.wo = w(q_out + 2 * kv_out, hidden), w(hidden, q_out)
        self.norm_w = torch.ones(hidden, dtype=torch.bfloat16, device=device)
        self.k_cache = torch.zeros(batch, acfg.n_kv_heads, acfg.max_seq, acfg.head_dim, dtype=torch.bfloat16, device=device)
        self.v_cache = torch.zeros_like(self.k_cache)

    def fill_cache(self, length: int, seed: int) -> None:
        """Stand-in for a prefill: random keys/values for the first ``length`` positions."""
        g = torch.Generator(device=self.k_cache.device).manual_seed(seed)
        self.k_cache[:, :, :length].copy_(torch.randn(self.k_cache[:, :, :length].shape, generator=g, device=self.k_cache.device) * 0.5)
        self.v_cache[:, :, :length].copy_(torch.randn(self.v_cache[:, :, :length].shape, generator=g, device=self.k_cache.device) * 0.5)

    def __call__(self, x: torch.Tensor, pos: torch.Tensor, mask: torch.Tensor) -> torch.Tensor:
        """``x [B, H]``; ``pos`` device int64 scalar (position being written); ``mask [1,1,1,max_seq]`` additive."""
        return x + self.delta(x, pos, mask)

    def delta(self, x: torch.Tensor, pos: torch.Tensor, mask: torch.Tensor) -> torch.Tensor:
        """What the attention adds to ``x``."""
        a = self.acfg
        h = _rmsnorm(x, self.norm_w, 1e-6)
        qkv = h @ self.wqkv.transpose(0, 1)
        q_out, kv_out = a.n_heads * a.head_dim, a.n_kv_heads * a.head_dim
        q = qkv[:, :q_out].view(self.batch, a.n_heads, 1, a.head_dim)
        k = qkv[:, q_out : q_out + kv_out].view(self.batch, a.n_kv_heads, 1, a.head_dim)
        v = qkv[:, q_out + kv_out :].view(self.batch, a.n_kv_heads, 1, a.head_dim)
        if qkv.is_cuda and qkv.dtype == torch.bfloat16 and a.head_dim % 8 == 0:
            from ..ops.kernels import kv_append

            kv_append(qkv[:, q_out : q_out + kv_out], qkv[:, q_out + kv_out :], self.k_cache, self.v_cache, pos)
        else:
            idx = pos.view(1, 1, 1, 1).expand(self.batch, a.n_kv_heads, 1, a.head_dim)
            self.k_cache.scatter_(2, idx, k)
            self.v_cache.scatter_(2, idx, v)
        o = F.scaled_dot_product_attention(q, self.k_cache, self.v_cache, attn_mask=mask, enable_gqa=True)
        return o.reshape(self.batch, q_out) @ self.wo.transpose(0, 1)


class DecodeModel:
    """``n_layers`` decoder layers for a fixed per-rank batch; ``step()`` runs one decode step from a graph."""

    def __init__(self, cfg: MoEConfig, rank: int, world: int, batch: int, n_layers: int, device, acfg: AttentionConfig | None = None,
                 group=None, seed: int = 0, attention: bool = True, weights_factory=None, fp8: bool = False,
                 own_router_gemm: bool = True):
        """``fp8``: the routed experts are kept as block-scaled e4m3 (one fp32 scale per 128x128 block, quantised
        from the random bf16 weights) and run on the ``kind::f8f6f4`` grouped GEMMs.  ``own_router_gemm``: router
        logits on the tcgen05 dense projection kernel instead of a library matmul."""
        self.cfg, self.rank, self.world, self.batch, self.device = cfg, rank, world, batch, torch.device(device)
        self.acfg = acfg or AttentionConfig()
        dev, H, I, L = self.device, cfg.hidden_size, cfg.moe_intermediate_size, cfg.experts_per_rank(world)
        g = torch.Generator(device=dev).manual_seed(seed * 7919 + rank)

        def randn(*shape, scale):
            return (torch.randn(*shape, generator=g, device=dev) * scale).to(torch.bfloat16)

        capacity = 1
        while capacity < batch:
            capacity *= 2
        # one set of communication buffers for all layers (they run one at a time)
        self.routed = FixedEPLayer(cfg, rank, world, None, None, capacity=capacity, group=group, device=dev, backend="cuda")
        self.layers = []
        for layer in range(n_layers):
            given = weights_factory(layer) if weights_factory is not None else None
            prequantised = given is not None and len(given) == 4  # (w13_q, w13_s, w2_q, w2_s): e4m3 + block scales
            if prequantised:
                w13 = w2 = None
            elif given is not None:
                w13, w2 = given
            else:
                w13 = torch.empty(L, 2 * I, H, dtype=torch.bfloat16, device=dev)
                w2 = torch.empty(L, H, I, dtype=torch.bfloat16, device=dev)
                for e in range(L):
                    w13[e] = randn(2 * I, H, scale=2.0 / math.sqrt(H))
                    w2[e] = randn(H, I, scale=1.0 / math.sqrt(I))
            pack = None
            if prequantised:
                pack = self.routed.make_fp8_pack(*given)
                maps = (None, None)
            elif fp8:
                from ..weights import quant_block_fp8

                def quantise(w):
                    qs, ss = zip(*(quant_block_fp8(w[e]) for e in range(w.shape[0])))
                    return torch.stack([q.view(torch.uint8) for q in qs]).view(torch.float8_e4m3fn), torch.stack(ss)

                q13, s13 = quantise(w13)
                q2, s2 = quantise(w2)
                pack = self.routed.make_fp8_pack(q13, s13, q2, s2)
                w13 = w2 = None  # only the e4m3 copies are kept
                maps = (None, None)
            else:
                maps = self.routed.make_weight_maps(w13, w2)
            gate_w = randn(cfg.n_routed_experts, H, scale=1.0 / math.sqrt(H)).to(torch.float32)
            router = RouterLogits(gate_w, capacity) if own_router_gemm else None
            bias = 0.05 * torch.randn(cfg.n_routed_experts, generator=g, device=dev)
            shared = None
            if cfg.n_shared_experts:
                Is = I * cfg.n_shared_experts
                shared = SharedExpert(randn(2 * Is, H, scale=2.0 / math.sqrt(H)), randn(H, Is, scale=1.0 / math.sqrt(Is)),
                                      capacity, cfg.swiglu_limit)
            norm_w = torch.ones(H, dtype=torch.bfloat16, device=dev)
            attn = Attention(H, self.acfg, batch, dev, seed * 31 + layer) if attention else None
            self.layers.append({"w13": w13, "w2": w2, "maps": maps, "fp8": pack, "gate_w": gate_w, "bias": bias,
                                "shared": shared, "norm_w": norm_w, "attn": attn, "router": router})
        self.x = torch.zeros(batch, H, dtype=torch.bfloat16, device=dev)
        self.out = torch.zeros_like(self.x)
        self.pos = torch.zeros((), dtype=torch.int64, device=dev)
        self.mask = torch.full((1, 1, 1, self.acfg.max_seq), float("-inf"), dtype=torch.bfloat16, device=dev)
        self.graph: torch.cuda.CUDAGraph | None = None
        self._side: torch.cuda.Stream | None = None  # warm-up before a capture, branches in it
        self._tail: torch.cuda.Stream | None = None  # the branch that moves the position on

    def prefill_standin(self, length: int) -> None:
        for i, layer in enumerate(self.layers):
            if layer["attn"] is not None:
                layer["attn"].fill_cache(length, 1000 + i)
        self.pos.fill_(length)
        self.mask.fill_(float("-inf"))
        self.mask[..., : length + 1] = 0

    def _forward(self, tail: torch.cuda.Stream | None = None) -> None:
        """``tail`` (captures only): a branch that moves the position on as soon as the last attention has used it, next to
        that layer's experts instead of behind them."""
        x = self.x
        for i, layer in enumerate(self.layers):
            delta = layer["attn"].delta(x, self.pos, self.mask) if layer["attn"] is not None else None
            if tail is not None and i == len(self.layers) - 1:
                tail.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(tail):
                    self._advance()
            if layer["fp8"] is not None:
                self.routed.bind_weights_fp8(layer["fp8"])
            else:
                self.routed.bind_weights(layer["w13"], layer["w2"], *layer["maps"])
            block = MoEBlock(self.cfg, self.routed, layer["gate_w"], layer["bias"], layer["norm_w"], layer["shared"],
                             router=layer["router"], branch=self._side)
            x = block(x, add=delta, out=self.out if i == len(self.layers) - 1 else None)
        if not self.layers:
            self.out.copy_(x)
        if tail is not None and self.layers:
            torch.cuda.current_stream().wait_stream(tail)

    def _advance(self) -> None:
        self.pos.add_(1)
        self.mask.view(-1).index_fill_(0, self.pos.view(1), 0.0)

    def capture(self) -> "DecodeModel":
        import torch.distributed as dist

        side = self._side = self._side or torch.cuda.Stream(device=self.device)
        self._tail = self._tail or torch.cuda.Stream(device=self.device)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            self._forward()
        torch.cuda.current_stream().wait_stream(side)
        torch.cuda.synchronize()
        if dist.is_available() and dist.is_initialized():
            dist.barrier()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self._forward(self._tail if self.layers else None)
            if not self.layers:
                self._advance()
        torch.cuda.synchronize()
        return self

    def step(self) -> torch.Tensor:
        """One decode step for the whole batch; advances the position (mask and KV write index)."""
        if self.graph is None:
            self._forward()
            self._advance()
        else:
            self.graph.replay()
        return self.out

    def check_status(self) -> dict:
        """The first status word that is set, of the routed experts and of every layer's router and shared expert: a wait that ran
        out leaves wrong values in the residual stream (device-to-host; call it between steps)."""
        from ..ops import _lib

        found = self.routed.check_status()
        for layer in self.layers:
            for part in (layer["router"], layer["shared"]):
                if found["code"] == 0 and getattr(part, "status", None) is not None:
                    found = _lib.decode_status(int(part.status.item()))
        return found

    def close(self) -> None:
        self.graph = None
