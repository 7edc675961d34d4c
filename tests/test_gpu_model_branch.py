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


@pytest.mark.parametrize("hidden,tokens,with_shared", [(4096, 1, True), (4096, 64, True), (4096, 65, True), (512, 64, True), (512, 64, False)])
def test_block_with_a_summand(hidden, tokens, with_shared):
    """`add`: normalisation and router logits in one launch or two (by size), eager and captured."""
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.models.glm_moe import MoEBlock, RouterLogits, SharedExpert
    from moeflow_b200.testing import make_bias, make_weights

    cfg = MoEConfig(hidden_size=hidden, moe_intermediate_size=256, n_routed_experts=36, n_shared_experts=int(with_shared), top_k=8)
    gen = torch.Generator().manual_seed(tokens)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    layer = FixedEPLayer(cfg, 0, 1, w13, w2, capacity=tokens, backend="cuda")
    gate = (torch.randn(36, hidden, generator=gen) / hidden**0.5).cuda()
    shared = SharedExpert((torch.randn(512, hidden, generator=gen) * 2 / hidden**0.5).bfloat16().cuda(),
                          (torch.randn(hidden, 256, generator=gen) / 16).bfloat16().cuda(), tokens, cfg.swiglu_limit) if with_shared else None
    router = RouterLogits(gate, tokens)
    gamma = (torch.rand(hidden, generator=gen) + 0.5).bfloat16().cuda()
    block = MoEBlock(cfg, layer, gate, make_bias(cfg, 1, device="cuda"), gamma, shared, router=router, branch=torch.cuda.Stream())
    x, add = (torch.zeros(tokens, hidden, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    out = torch.empty_like(x)
    block(x, add=add, out=out)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        block(x, add=add, out=out)
    for _ in range(5):
        for t in (x, add):
            t.copy_(torch.randn(tokens, hidden, generator=gen).bfloat16())
        graph.replay()
        got, captured = out.clone(), router.logits.clone()
        assert torch.equal(got, block(x, add=add, out=torch.empty_like(x))) and torch.equal(captured, router.logits)
        total = (x + add).double()
        h = (total * torch.rsqrt(total.pow(2).mean(-1, keepdim=True) + 1e-6) * gamma.double()).bfloat16().double()
        exact = h @ router.w[:36].double().t()
        # h is rounded to bf16 from fp32 there and from fp64 here: single values differ by a rounding step, 2**-8 of them at most; the
        # fp32 sums err by hidden * 2**-24 of the absolute sum
        assert bool(((captured.double() - exact).abs() <= (2.0**-8 + hidden * 2.0**-24) * (h.abs() @ router.w[:36].double().abs().t())).all())
    assert layer.check_status()["code"] == 0 and int(router.status) == 0
