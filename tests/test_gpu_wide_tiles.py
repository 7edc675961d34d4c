"""256-row token tiles that hold few rows next to full ones: units of up to 128 token columns take one accumulator stage,
wider ones both, in any order.  Against the layer with 64-row tiles and float64 experts."""

import pytest
import torch

from moeflow_b200 import MoEConfig
from moeflow_b200.testing import make_hidden, make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("inter", [128, 384])
@pytest.mark.parametrize("counts", [(1, 256, 16, 129, 128, 0, 257, 63), (128,) * 8, (129,) * 8, (300, 5, 300, 5, 64, 65, 192, 193)])
def test_narrow_and_wide_units(counts, inter):
    from moeflow_b200.fixed import FixedEPLayer

    cfg = MoEConfig(hidden_size=512, moe_intermediate_size=inter, n_routed_experts=8, top_k=1)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    t = sum(counts)
    x = make_hidden(t, cfg, 1, device="cuda")
    g = torch.Generator().manual_seed(2)
    ids = torch.repeat_interleave(torch.arange(8), torch.tensor(counts))[torch.randperm(t, generator=g)].int()[:, None].cuda()
    weights = torch.rand(t, 1, generator=g).cuda() + 0.5
    outs = {}
    for block_m in (64, 256):
        layer = FixedEPLayer(cfg, 0, 1, w13, w2, capacity=t, backend="cuda", gemm_kwargs={"block_m": block_m}, wait_ns=100_000_000)
        outs[block_m] = layer.forward_routed(x, weights, ids).clone()
        assert torch.equal(layer.forward_routed(x, weights, ids), outs[block_m])
        assert layer.check_status()["code"] == 0
    exact = torch.empty(t, 512, dtype=torch.float64, device="cuda")
    for e in range(8):
        rows = ids[:, 0] == e
        h = x[rows].double() @ w13[e].double().t()
        gate, up = h[:, :inter], h[:, inter:]
        if cfg.swiglu_limit is not None:
            gate, up = gate.clamp(max=cfg.swiglu_limit), up.clamp(-cfg.swiglu_limit, cfg.swiglu_limit)
        exact[rows] = weights[rows].double() * ((torch.nn.functional.silu(gate) * up) @ w2[e].double().t())
    for out in outs.values():
        # activations and result are rounded to bf16 once each (2**-9 of a value at most, averaged over a row)
        err = (out.double() - exact).norm(dim=1) / exact.norm(dim=1)
        assert float(err.max()) < 2 * 2.0**-8


@pytest.mark.parametrize("K", [128, 384, 1536, 2048, 4096])
def test_expansion_is_exact(K):
    from moeflow_b200.ops.fp8 import expand_block_fp8

    g = torch.Generator().manual_seed(K)
    w = torch.randn(256, K, generator=g).to(torch.float8_e4m3fn).cuda()
    s = torch.rand(2, K // 128, generator=g).cuda() + 0.1
    want = (w.float() * s.repeat_interleave(128, 0).repeat_interleave(128, 1)).bfloat16()
    assert torch.equal(expand_block_fp8(w, s), want)


@pytest.mark.parametrize("tokens", [1, 3, 8, 100])
@pytest.mark.parametrize("experts", [8, 36, 288])
def test_k_splits_of_the_one_pass_metadata(tokens, experts):
    """The splits weighed by four lanes are those of the host's cost model."""
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.ops import _lib
    from moeflow_b200.testing import make_logits

    cfg = MoEConfig(hidden_size=512, moe_intermediate_size=256, n_routed_experts=experts, top_k=4)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    layer = FixedEPLayer(cfg, 0, 1, w13, w2, capacity=tokens, backend="cuda")
    layer.forward(make_hidden(tokens, cfg, 1, device="cuda"), make_logits(tokens, cfg, 2, device="cuda"), None, stop_after="META")
    plan = layer.plan.tolist()
    cols = max(16, (int(layer.tile_n[: plan[0]].max()) + 15) // 16 * 16)
    floats = layer._a_meta.partial_floats
    for word, m, k, per, over in ((1, 2, 8, 256, 4), (2, 4, 4, 128, 8)):
        want = _lib.lib().mf_plan_split(plan[0] * m, k, layer.n_sms, floats // (per * cols), over, cols)
        assert plan[word] == want


@pytest.mark.parametrize("hidden,inter,tokens", [(512, 256, 600), (768, 128, 300), (512, 384, 90), (4096, 1536, 600)])
def test_down_weights_expanded_beside_the_gate_up_gemm(hidden, inter, tokens):
    """The same bits as with both expansions ahead of the GEMMs; weights that change between forwards are expanded anew."""
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.testing import make_bias, make_logits
    from moeflow_b200.weights import quant_block_fp8

    cfg = MoEConfig(hidden_size=hidden, moe_intermediate_size=inter, n_routed_experts=4, top_k=2)
    bias = make_bias(cfg, 1, device="cuda")
    layers = [FixedEPLayer(cfg, 0, 1, None, None, capacity=tokens, device="cuda", backend="cuda", wait_ns=200_000_000,
                           gemm_kwargs={"block_m": 256, "permute_rows": False, "expand_beside": beside}) for beside in (True, False)]
    for seed in range(3):
        def pack(w):
            q, s = zip(*(quant_block_fp8(m) for m in w))
            return torch.stack([t.view(torch.uint8) for t in q]).view(torch.float8_e4m3fn).cuda(), torch.stack(list(s)).cuda()

        w13, w2 = make_weights(cfg, seed, dtype=torch.float32)
        weights = (*pack(w13), *pack(w2))
        x, lg = make_hidden(tokens, cfg, 10 + seed, device="cuda"), make_logits(tokens, cfg, 20 + seed, device="cuda")
        outs = []
        for layer in layers:
            layer.set_weights_fp8(*weights)
            FixedEPLayer._expand_scratch[(layer.device.index, layer.L, layer.I, layer.H)]["w2"].fill_(float("nan"))
            outs.append(layer.forward(x, lg, bias)[:tokens].clone())
            assert layer.check_status()["code"] == 0
        assert bool(torch.isfinite(outs[0].float()).all()) and outs[0].abs().sum() > 0 and torch.equal(*outs)


def test_an_empty_forward_ends_behind_the_expansion_beside_it():
    """No token tile: the down GEMM waits for no tile and no weights, but the call is over only when its gate/up GEMM has expanded
    everything, since the next layer on these buffers sets the counter back and writes to the same scratch."""
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.testing import make_bias, make_logits

    cfg = MoEConfig(hidden_size=4096, moe_intermediate_size=1536, n_routed_experts=8, top_k=2)
    layer = FixedEPLayer(cfg, 0, 1, None, None, capacity=300, device="cuda", backend="cuda", wait_ns=200_000_000,
                         gemm_kwargs={"block_m": 256, "permute_rows": False, "expand_beside": True})

    def pack(seed):
        g = torch.Generator(device="cuda").manual_seed(seed)
        q = [(torch.randn(*s, generator=g, device="cuda")).to(torch.float8_e4m3fn) for s in ((8, 3072, 4096), (8, 4096, 1536))]
        s = [torch.rand(*s, generator=g, device="cuda") * 0.02 + 0.001 for s in ((8, 24, 32), (8, 32, 12))]
        return layer.make_fp8_pack(q[0], s[0], q[1], s[1])

    packs = [pack(seed) for seed in (1, 2, 3)]
    x, lg, bias = make_hidden(300, cfg, 4, device="cuda"), make_logits(300, cfg, 5, device="cuda"), make_bias(cfg, 6, device="cuda")
    none, done, outs = torch.zeros((), dtype=torch.int32, device="cuda"), [], []

    def calls():
        done.clear(), outs.clear()
        for i, p in enumerate(packs):
            layer.bind_weights_fp8(p)
            empty = layer.forward(x, lg, bias, none)
            done.append(layer._expand_done.clone())
            outs.append(empty.clone())
            layer.bind_weights_fp8(packs[(i + 1) % 3])
            outs.append(layer.forward(x, lg, bias).clone())

    calls()
    want = [o.clone() for o in outs]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        calls()
    for _ in range(5):
        graph.replay()
        torch.cuda.synchronize()
        assert [int(d) for d in done] == [packs[0]["w2"].numel() // 4096] * 3
        for got, right in zip(outs, want):
            assert torch.equal(got, right)
        assert not outs[0].any() and bool(outs[1].any())
    assert layer.check_status()["code"] == 0
