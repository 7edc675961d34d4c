"""The stages of one rank called one by one: weights bound, rows rewritten or a graph captured between the dispatch and
the experts.  Every order must give bitwise what the whole forward gives, in which the dispatch launch also builds the
metadata and quantises the rows."""

import pytest
import torch

from moeflow_b200 import MoEConfig
from moeflow_b200.testing import make_bias, make_hidden, make_logits, make_weights
from moeflow_b200.weights import quant_block_fp8

pytestmark = pytest.mark.gpu

CFG = MoEConfig(hidden_size=512, moe_intermediate_size=256, n_routed_experts=8, top_k=2)
TOKENS, CAPACITY = 13, 16


@pytest.fixture(scope="module")
def weights():
    w13, w2 = make_weights(CFG, 0, device="cuda")
    quantised = [[quant_block_fp8(w[e].float()) for e in range(CFG.n_routed_experts)] for w in (w13, w2)]
    packs = []
    for pairs in quantised:
        packs += [torch.stack([q.view(torch.uint8) for q, _ in pairs]).view(torch.float8_e4m3fn), torch.stack([s for _, s in pairs])]
    return (w13, w2), tuple(packs)


def _layer():
    from moeflow_b200.fixed import FixedEPLayer

    return FixedEPLayer(CFG, 0, 1, None, None, capacity=CAPACITY, device=torch.device("cuda", 0), backend="cuda",
                        gemm_kwargs={"fp8_weights": False}, wait_ns=50_000_000)


def _bind(layer, weights, kind):
    if kind == "bf16":
        layer.set_weights(*weights[0])
    elif kind == "e4m3":
        layer.set_weights_fp8(*weights[1])


def _inputs(seed):
    return make_hidden(TOKENS, CFG, seed, device="cuda"), make_logits(TOKENS, CFG, seed + 9, device="cuda")


def _whole(weights, kind, seed):
    layer = _layer()
    assert layer.fuse_meta
    _bind(layer, weights, kind)
    out = layer.forward(*_inputs(seed), make_bias(CFG, 1, device="cuda")).clone()
    assert layer.check_status()["code"] == 0
    return out


@pytest.mark.parametrize("before", ["none", "bf16", "e4m3"])
@pytest.mark.parametrize("after", ["bf16", "e4m3"])
def test_weights_bound_between_dispatch_and_experts(weights, before, after):
    layer, bias = _layer(), make_bias(CFG, 1, device="cuda")
    _bind(layer, weights, before)
    for seed in (1, 2):  # the second time another forward's rows are in the buffers
        hit = layer.stage_pack(*_inputs(seed), bias)
        _bind(layer, weights, after)
        layer.stage_experts()
        assert torch.equal(layer.stage_combine(hit, torch.bfloat16), _whole(weights, after, seed))
    assert layer.check_status()["code"] == 0


@pytest.mark.parametrize("kind", ["bf16", "e4m3"])
def test_rows_rewritten_and_experts_captured_alone(weights, kind):
    layer, bias = _layer(), make_bias(CFG, 1, device="cuda")
    _bind(layer, weights, kind)
    layer.forward(*_inputs(2), bias, stop_after="DISPATCH")
    rows = layer._recv_store.clone()
    hit = layer.stage_pack(*_inputs(1), bias)
    layer._recv_store.copy_(rows)
    layer.stage_experts()
    assert torch.equal(layer.stage_combine(hit, torch.bfloat16), _whole(weights, kind, 2))

    layer.forward(*_inputs(1), bias, stop_after="A2A_FORWARD")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        layer.stage_experts()
    for seed in (3, 4):
        hit = layer.stage_pack(*_inputs(seed), bias)
        graph.replay()
        assert torch.equal(layer.stage_combine(hit, torch.bfloat16), _whole(weights, kind, seed))
    assert layer.check_status()["code"] == 0


def test_experts_run_twice_on_one_dispatch(weights):
    layer, bias = _layer(), make_bias(CFG, 1, device="cuda")
    _bind(layer, weights, "e4m3")
    hit = layer.stage_pack(*_inputs(1), bias)
    for kind in ("e4m3", "bf16", "e4m3"):
        _bind(layer, weights, kind)
        layer.stage_experts()
        assert torch.equal(layer.stage_combine(hit, torch.bfloat16), _whole(weights, kind, 1))
