"""MoE block whose shared expert starts on a branch of the captured graph: same numbers as the eager block, step after step,
with inputs that change between replays."""

import pytest
import torch

from moeflow_b200 import MoEConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tokens", [1, 7, 64])
def test_captured_block_equals_the_eager_one(tokens):
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.models.glm_moe import MoEBlock, RouterLogits, SharedExpert
    from moeflow_b200.testing import make_bias, make_weights

    cfg = MoEConfig(hidden_size=512, moe_intermediate_size=256, n_routed_experts=16, n_shared_experts=1, top_k=4)
    gen = torch.Generator().manual_seed(tokens)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    layer = FixedEPLayer(cfg, 0, 1, w13, w2, capacity=tokens, backend="cuda")
    gate = (torch.randn(16, 512, generator=gen) / 512**0.5).cuda()
    shared = SharedExpert((torch.randn(512, 512, generator=gen) * 2 / 512**0.5).bfloat16().cuda(),
                          (torch.randn(512, 256, generator=gen) / 16).bfloat16().cuda(), tokens, cfg.swiglu_limit)
    block = MoEBlock(cfg, layer, gate, make_bias(cfg, 1, device="cuda"), torch.ones(512, dtype=torch.bfloat16, device="cuda"), shared,
                     router=RouterLogits(gate, tokens), branch=torch.cuda.Stream())
    x = torch.zeros(tokens, 512, dtype=torch.bfloat16, device="cuda")
    out = torch.empty_like(x)
    block(x, out=out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        block(x, out=out)
    for _ in range(20):
        x.copy_(torch.randn(tokens, 512, generator=gen).bfloat16())
        graph.replay()
        got = out.clone()
        assert torch.equal(got, block(x, out=torch.empty_like(x)))
    assert layer.check_status()["code"] == 0 and int(shared.status) == 0


@pytest.mark.parametrize("tokens", [3, 16])
def test_captured_block_into_rows_that_the_last_kernel_does_not_write(tokens):
    """Outputs off the 16-byte grid, with rows behind those of the step, or with a pitch: what the down projection stores."""
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.models.glm_moe import MoEBlock, RouterLogits, SharedExpert
    from moeflow_b200.testing import make_bias, make_weights

    cfg = MoEConfig(hidden_size=512, moe_intermediate_size=256, n_routed_experts=16, n_shared_experts=1, top_k=4)
    gen = torch.Generator().manual_seed(tokens)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    layer = FixedEPLayer(cfg, 0, 1, w13, w2, capacity=tokens, backend="cuda")
    gate = (torch.randn(16, 512, generator=gen) / 512**0.5).cuda()
    shared = SharedExpert((torch.randn(512, 512, generator=gen) * 2 / 512**0.5).bfloat16().cuda(),
                          (torch.randn(512, 256, generator=gen) / 16).bfloat16().cuda(), tokens, cfg.swiglu_limit)
    block = MoEBlock(cfg, layer, gate, make_bias(cfg, 1, device="cuda"), torch.ones(512, dtype=torch.bfloat16, device="cuda"), shared,
                     router=RouterLogits(gate, tokens), branch=torch.cuda.Stream())
    x = torch.randn(tokens, 512, generator=gen).bfloat16().cuda()
    want = block(x).clone()
    store = [torch.full((tokens * 512 + 8,), 7.0, dtype=torch.bfloat16, device="cuda"),
             torch.full((tokens + 5, 512), 7.0, dtype=torch.bfloat16, device="cuda"),
             torch.full((tokens, 1024), 7.0, dtype=torch.bfloat16, device="cuda")]
    outs = [store[0][1 : 1 + tokens * 512].view(tokens, 512), store[1], store[2][:, 128:640]]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [block(x, out=out) for out in outs]
    graph.replay()
    for g, out in zip(got, outs):
        assert g.shape == want.shape and torch.equal(g, want) and torch.equal(out[:tokens], want)
    assert bool((store[0][0] == 7).all()) and bool((store[0][1 + tokens * 512 :] == 7).all()) and bool((store[1][tokens:] == 7).all())
    assert bool((store[2][:, :128] == 7).all()) and bool((store[2][:, 640:] == 7).all())
    assert layer.check_status()["code"] == 0 and int(shared.status) == 0
