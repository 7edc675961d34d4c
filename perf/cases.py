"""The workloads this framework is timed on, as its users run them: one routed MoE layer (or one decoder layer of
the serving model) per pass, from single-token decode calls to long prefills.

The layer shape is GLM-5.3-Flash (hidden 4096, top-8, sigmoid routing with a selection bias) with expert intermediate
size 1536 (the benchmark shape) or 2048 (the checkpoint's), and the small generic layer of the command-line smoke
runs.  ``experts`` is the number of experts on this GPU: all 288 of a layer, or a rank's share of an expert-parallel
group (144, 72, 36 for 2, 4, 8 ranks).  Expert weights are bf16, or e4m3 with 128x128 block scales (the FP8
checkpoint).  Five ways of calling:

    graph    ``GraphedMoELayer(x, logits)``: a decode step's layer call, inputs on the device
    pinned   ``GraphedMoELayer.step(block, out)``: the same call fed from and read back to pinned host memory
    eager    ``FixedEPLayer.forward``: a prefill chunk
    routed   ``FixedEPLayer.forward_routed``: the serving engine's call, which has routed the tokens itself
    model    ``DecodeModel.step``: attention, router, routed and shared experts of one decoder layer, one token per
             sequence
"""

from __future__ import annotations

import dataclasses
import math

import torch

from moeflow_b200.config import GLM53_FLASH, MoEConfig
from moeflow_b200.fixed import FixedEPLayer
from moeflow_b200.models.glm_moe import AttentionConfig, DecodeModel
from moeflow_b200.models.routed_moe import GraphedMoELayer
from moeflow_b200.ops.kernels import router_topk
from moeflow_b200.testing import make_bias, make_logits
from moeflow_b200.weights import quant_block_fp8

#: Decode steps after which the model's sequences start again (the length of one answer).
ANSWER = 512


def _case(name, kind, tokens, capacity, experts, weights="bf16", inter=1536, dist="uniform", context=0):
    return {"name": name, "kind": kind, "shape": "glm", "tokens": tokens, "capacity": capacity, "experts": experts,
            "inter": inter, "weights": weights, "dist": dist, "context": context}


def listed():
    return [
        # The generic small layer (hidden 512, intermediate 256, 32 experts, top-4): nothing but launch and
        # synchronisation latency.
        {"name": "small layer, 8 tokens", "kind": "graph", "shape": "small", "tokens": 8, "capacity": 8, "experts": 32,
         "inter": 256, "weights": "bf16", "dist": "uniform", "context": 0},
        # One user, one token at a time, all experts of the layer on this GPU.
        _case("decode 1, bf16, 288 experts", "graph", 1, 1, 288),
        # A few users on the FP8 checkpoint.
        _case("decode 8, e4m3, 288 experts", "graph", 8, 8, 288, "e4m3"),
        # A serving process that hands over host buffers; 24 live rows in the 32-row graph; a rank of 4.
        _case("decode 24 of 32, host, bf16", "pinned", 24, 32, 72),
        # The headline benchmark: 128 tokens on the whole layer.
        _case("decode 128, bf16, 288 experts", "graph", 128, 128, 288),
        # Skewed popularity on a rank of 8, ragged batch, FP8 checkpoint.
        _case("decode 100 zipf, e4m3", "graph", 100, 128, 36, "e4m3", dist="zipf"),
        # The engine's call for a mixed batch (decodes and a piece of a prefill), checkpoint intermediate size.
        _case("engine 250, e4m3, inter 2048", "routed", 250, 256, 72, "e4m3", inter=2048),
        # A prefill of one ordinary prompt on a rank of 4.
        _case("prefill 1000, bf16", "eager", 1000, 1024, 72),
        # A chunk of a chunked prefill, FP8 checkpoint, a rank of 8.
        _case("prefill 2000, e4m3", "eager", 2000, 2048, 36, "e4m3"),
        # The long-prefill configuration: 8192 tokens, FP8 checkpoint, a rank of 8.
        _case("prefill 8192, e4m3", "eager", 8192, 8192, 36, "e4m3"),
        # Whole decoder layers inside a decode step: low and high concurrency at 1024 tokens of context.
        _case("model 4 sequences, bf16", "model", 4, 4, 36, context=1024),
        _case("model 64 sequences, e4m3", "model", 64, 64, 36, "e4m3", context=1024),
    ]


def _spread(rng, low, high):
    """A whole number, log-uniform between the bounds."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def _bucket(rng, tokens):
    """Graph capacities are powers of two in a serving process, or exactly the batch in a fixed-size job."""
    return tokens if rng.random() < 0.3 else 1 << (tokens - 1).bit_length()


def draw(rng):
    kind = rng.choices(("graph", "pinned", "eager", "routed", "model"), (6, 2, 5, 3, 4))[0]
    weights = rng.choice(("bf16", "e4m3"))
    inter = rng.choice((1536, 1536, 2048))
    dist = rng.choice(("uniform", "uniform", "zipf"))
    context = 0
    if kind in ("graph", "pinned"):
        if rng.random() < 0.1:
            t = _spread(rng, 1, 128)
            return {"kind": kind, "shape": "small", "tokens": t, "capacity": _bucket(rng, t), "experts": 32, "inter": 256,
                    "weights": "bf16", "dist": dist, "context": 0}
        experts = rng.choice((36, 72, 144, 288))
        inter = 1536
        tokens = _spread(rng, 1, 128)
    elif kind == "eager":
        experts = rng.choice((36, 72))
        tokens = _spread(rng, 129, 8192 if inter == 1536 and experts == 36 else 5000)
    elif kind == "routed":
        experts = rng.choice((36, 72, 144))
        tokens = _spread(rng, 1, 1024)
    else:
        experts = rng.choice((36, 72))
        tokens = _spread(rng, 1, 64)
        context = _spread(rng, 128, 1024)
        dist = "uniform"
    capacity = _bucket(rng, tokens)
    if kind == "model":
        capacity = 1 << (tokens - 1).bit_length()
    return {"kind": kind, "shape": "glm", "tokens": tokens, "capacity": capacity, "experts": experts, "inter": inter,
            "weights": weights, "dist": dist, "context": context}


# ---- inputs ---------------------------------------------------------------------------------------------
def _config(case) -> MoEConfig:
    if case["shape"] == "small":
        return MoEConfig(hidden_size=512, moe_intermediate_size=case["inter"], n_routed_experts=case["experts"], top_k=4)
    return dataclasses.replace(GLM53_FLASH, moe_intermediate_size=case["inter"], n_routed_experts=case["experts"])


def _expert_weights(cfg: MoEConfig, e4m3: bool, gen: torch.Generator):
    """Random-init experts, activations O(1): ``(w13, w2)`` bf16 or ``(w13, scales, w2, scales)`` e4m3."""
    n, H, I = cfg.n_routed_experts, cfg.hidden_size, cfg.moe_intermediate_size

    def dense(rows, cols, std):
        w = torch.empty(n, rows, cols, dtype=torch.bfloat16, device="cuda")
        for e in range(n):
            w[e].normal_(0.0, std, generator=gen)
        return w

    def blocks(rows, cols, std):
        q = torch.empty(n, rows, cols, dtype=torch.float8_e4m3fn, device="cuda")
        s = torch.empty(n, rows // 128, cols // 128, dtype=torch.float32, device="cuda")
        for e in range(n):
            q[e], s[e] = quant_block_fp8(torch.empty(rows, cols, device="cuda").normal_(0.0, std, generator=gen))
        return q, s

    make = blocks if e4m3 else dense
    first, second = make(2 * I, H, 2.0 / math.sqrt(H)), make(H, I, 1.0 / math.sqrt(I))
    return (*first, *second) if e4m3 else (first, second)


def _tokens(case, cfg: MoEConfig, seed: int, gen: torch.Generator):
    """``(hidden rows, router logits, selection bias)`` on the GPU."""
    x = torch.randn(case["tokens"], cfg.hidden_size, generator=gen, device="cuda").to(torch.bfloat16)
    return x, make_logits(case["tokens"], cfg, seed + 7, dist=case["dist"], device="cuda"), make_bias(cfg, seed + 1, device="cuda")


def _layer(cfg: MoEConfig, capacity: int, weights) -> FixedEPLayer:
    device = torch.device("cuda", torch.cuda.current_device())
    if len(weights) == 2:
        return FixedEPLayer(cfg, 0, 1, *weights, capacity=capacity, backend="cuda")
    layer = FixedEPLayer(cfg, 0, 1, None, None, capacity=capacity, device=device, backend="cuda")
    layer.set_weights_fp8(*weights)
    return layer


def prepare(case, seed):
    cfg, kind = _config(case), case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    weights = _expert_weights(cfg, case["weights"] == "e4m3", gen)
    if kind == "model":
        device = torch.device("cuda", torch.cuda.current_device())
        heads = AttentionConfig(max_seq=case["context"] + ANSWER + 8)
        # One layer: a deeper stack repeats it, and with more of them the rounding of one layer's sum may tip the
        # expert choice of a later one, so that no tolerance could be stated.
        model = DecodeModel(cfg, 0, 1, case["tokens"], 1, device, heads, seed=seed, weights_factory=lambda layer: weights,
                            fp8=case["weights"] == "e4m3")
        model.prefill_standin(case["context"])
        x = torch.randn(case["tokens"], cfg.hidden_size, generator=gen, device="cuda").to(torch.bfloat16)
        model.x.copy_(x)
        model.capture()
        return {"kind": kind, "model": model, "x": x, "context": case["context"], "steps": 0}
    layer = _layer(cfg, case["capacity"], weights)
    x, logits, bias = _tokens(case, cfg, seed, gen)
    state = {"kind": kind, "layer": layer, "x": x, "logits": logits, "bias": bias}
    if kind in ("graph", "pinned"):
        state["step"] = GraphedMoELayer(layer, bias).capture()
    if kind == "pinned":
        block = state["step"].new_pinned_inputs()
        block.x[: case["tokens"]].copy_(x)
        block.logits[: case["tokens"]].copy_(logits)
        block.set_rows(case["tokens"])
        state["block"] = block
        state["out"] = torch.zeros(case["tokens"], cfg.hidden_size, dtype=torch.bfloat16).pin_memory()
    if kind == "routed":
        state["weights"], state["ids"] = router_topk(logits, bias, cfg)
    return state


# ---- one pass -------------------------------------------------------------------------------------------
def run(state):
    kind = state["kind"]
    if kind == "graph":
        return state["step"](state["x"], state["logits"])
    if kind == "pinned":
        return state["step"].step(state["block"], state["out"])
    if kind == "eager":
        return state["layer"].forward(state["x"], state["logits"], state["bias"])[: state["x"].shape[0]]
    if kind == "routed":
        return state["layer"].forward_routed(state["x"], state["weights"], state["ids"])
    model = state["model"]
    if state["steps"] == ANSWER:  # every sequence is answered: the next ones start from their prompts
        model.pos.fill_(state["context"])
        model.mask[..., state["context"] + 1 :] = float("-inf")
        state["steps"] = 0
    state["steps"] += 1
    model.x.copy_(state["x"])  # this step's embedded tokens
    return model.step()


# ---- what a pass cannot do without ------------------------------------------------------------------------
def _active_experts(case, cfg: MoEConfig) -> int:
    """Experts that at least one token chooses, from a sample of the case's routing."""
    logits = make_logits(case["tokens"], cfg, 7, dist=case["dist"])
    chosen = (torch.sigmoid(logits) + make_bias(cfg, 1)).topk(cfg.top_k, dim=-1).indices
    return int(chosen.unique().numel())


def work(case):
    cfg, t = _config(case), case["tokens"]
    H, I, E = cfg.hidden_size, cfg.moe_intermediate_size, cfg.n_routed_experts
    width = 1 if case["weights"] == "e4m3" else 2
    nbytes = _active_experts(case, cfg) * 3 * H * I * width + 2 * t * H * 2
    flops = 2 * t * cfg.top_k * 3 * H * I
    if case["kind"] == "model":
        a, length = AttentionConfig(), case["context"] + ANSWER // 2
        q, kv = a.n_heads * a.head_dim, a.n_kv_heads * a.head_dim
        dense = H * (q + 2 * kv) + q * H + E * H + 3 * H * I * cfg.n_shared_experts  # attention, router, shared expert
        nbytes += 2 * dense + 2 * t * length * kv * 2
        flops += 2 * t * dense + 4 * t * length * q
    else:
        nbytes += 8 * t * cfg.top_k if case["kind"] == "routed" else 4 * t * E
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """bf16 tensors with fp32 sums in between: activations, expert rows and the layer's output are each rounded to
    bf16 once (2**-9 relative), and a sum in another order may move any of these roundings."""
    return {"rel": 1e-2}
