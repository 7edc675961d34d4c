"""Layers built for bf16 weights at 36 to 80 expected rows per expert, bound to e4m3 weights and back: every weight type has the tile
height and the kernels that it has in a layer of its own, bit for bit."""

import pytest
import torch

from moeflow_b200 import MoEConfig
from moeflow_b200.testing import make_bias, make_hidden, make_logits, make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("built_with_weights", [True, False])
@pytest.mark.parametrize("experts,tokens,bf16_rows", [(36, 200, 256), (8, 72, 256), (8, 40, 64)])
def test_e4m3_weights_on_a_layer_built_for_bf16(experts, tokens, bf16_rows, built_with_weights):
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.weights import quant_block_fp8

    cfg = MoEConfig(hidden_size=512, moe_intermediate_size=256, n_routed_experts=experts, top_k=8)
    w13, w2 = make_weights(cfg, 0, device="cuda")

    def quantise(w):
        q, s = zip(*(quant_block_fp8(m) for m in w.float().cpu()))
        return torch.stack([t.view(torch.uint8) for t in q]).view(torch.float8_e4m3fn).cuda(), torch.stack(list(s)).cuda()

    e4m3 = (*quantise(w13), *quantise(w2))
    x, lg, bias = make_hidden(tokens, cfg, 1, device="cuda"), make_logits(tokens, cfg, 2, device="cuda"), make_bias(cfg, 3, device="cuda")

    def make(weights, **kw):
        return FixedEPLayer(cfg, 0, 1, *weights, capacity=tokens, device="cuda", backend="cuda", gemm_kwargs=kw, wait_ns=200_000_000)

    def run(layer, rows):
        out = layer.forward(x, lg, bias)[:tokens].clone()
        again = layer.forward(x, lg, bias)[:tokens]
        assert layer.check_status()["code"] == 0 and layer.block_m == rows and torch.equal(out, again) and out.abs().sum() > 0
        return out

    want_bf16 = run(make((w13, w2), block_m=bf16_rows, permute_rows=False), bf16_rows)
    own = make((None, None), block_m=128)
    own.set_weights_fp8(*e4m3)
    want_e4m3 = run(own, 128)
    FixedEPLayer.release_expand_scratch()
    layer = make((w13, w2) if built_with_weights else (None, None), **({} if built_with_weights else {"fp8_weights": False}))
    pack = layer.make_fp8_pack(*e4m3)
    assert "expand" not in pack
    for _ in range(2):
        layer.bind_weights_fp8(pack)
        assert torch.equal(run(layer, 128), want_e4m3)
        layer.set_weights(w13, w2)
        assert torch.equal(run(layer, bf16_rows), want_bf16)
    assert not FixedEPLayer._expand_scratch  # no bf16 copy of the experts
    # forwards of both kinds in one graph, on the same buffers
    outs = []
    maps = layer.make_weight_maps(w13, w2)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(2):
            layer.bind_weights_fp8(pack)
            outs.append(layer.forward(x, lg, bias)[:tokens].clone())
            layer.bind_weights(w13, w2, *maps)
            outs.append(layer.forward(x, lg, bias)[:tokens].clone())
    for _ in range(3):
        graph.replay()
        assert all(torch.equal(o, w) for o, w in zip(outs, (want_e4m3, want_bf16) * 2)) and layer.check_status()["code"] == 0


def test_a_given_height_holds_for_both_types():
    from moeflow_b200.fixed import FixedEPLayer

    cfg = MoEConfig(hidden_size=512, moe_intermediate_size=256, n_routed_experts=8, top_k=8)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    q13, q2 = (torch.zeros(w.shape, dtype=torch.uint8, device="cuda").view(torch.float8_e4m3fn) for w in (w13, w2))
    scales = torch.ones(8, 4, 4, device="cuda"), torch.ones(8, 4, 2, device="cuda")
    for rows in (32, 64, 128, 256):
        layer = FixedEPLayer(cfg, 0, 1, w13, w2, capacity=64, backend="cuda", gemm_kwargs={"block_m": rows})
        pack = layer.make_fp8_pack(q13, scales[0], q2, scales[1])
        assert bool(pack.get("expand")) == (rows == 256)
        layer.bind_weights_fp8(pack)
        assert layer.block_m == rows
