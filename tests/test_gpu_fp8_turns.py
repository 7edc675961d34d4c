"""e4m3 gate/up GEMM on 64-row tiles: the two promotion groups take narrow units in turn, wide ones together."""

import pytest
import torch

from moeflow_b200 import MoEConfig
from moeflow_b200.testing import make_bias, make_hidden, make_logits, make_weights
from moeflow_b200.tolerances import normwise_rel_err
from moeflow_b200.weights import dequant_block_fp8, quant_block_fp8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,split", [(128, 1), (256, 1), (256, 2), (768, 1), (1024, 2), (768, 0)])
@pytest.mark.parametrize("grid", [1, 2, None])
def test_narrow_and_wide_units_in_any_order(hidden, split, grid):
    """One CTA that does every unit, units shorter than the accumulators ahead (1 to 4 K blocks), cut units."""
    from moeflow_b200.ops.fp8 import dequant_rows, gate_up_swiglu_fp8, quant_rows_1x128
    from moeflow_b200.ops.grouped_gemm import plan_from_offsets

    counts, inter = [1, 32, 33, 16, 64, 64, 20, 2, 31, 48], 128
    gen = torch.Generator().manual_seed(hidden)
    packs = [quant_block_fp8(torch.randn(2 * inter, hidden, generator=gen) * (2.0 / hidden**0.5)) for _ in counts]
    w = torch.stack([q.view(torch.uint8) for q, _ in packs]).view(torch.float8_e4m3fn).cuda()
    s = torch.stack([s for _, s in packs]).cuda()
    n = sum(counts)
    offsets = [sum(counts[:i]) for i in range(len(counts) + 1)]
    xq, xs = quant_rows_1x128(torch.randn(n, hidden, generator=gen).bfloat16().cuda())
    status = torch.zeros(1, dtype=torch.int64, device="cuda")
    tp = plan_from_offsets(offsets, 64, xq.device)
    act = gate_up_swiglu_fp8(xq, xs, w, s, tp, limit=10.0, split=split, grid=grid, status=status, wait_ns=50_000_000)
    assert int(status) == 0
    x = dequant_rows(xq, xs)
    for e, (lo, hi) in enumerate(zip(offsets[:-1], offsets[1:])):
        gate, up = (x[lo:hi] @ dequant_block_fp8(w[e], s[e]).t()).chunk(2, dim=-1)
        ref = torch.nn.functional.silu(gate.clamp(max=10.0)) * up.clamp(-10.0, 10.0)
        # one bf16 rounding of every element (2**-9) on sums whose fp32 error is far below it
        assert normwise_rel_err(act[lo:hi], ref) < 4 * 2.0**-8


@pytest.mark.parametrize("tokens", [1, 20, 64])
def test_layer_bits_do_not_depend_on_who_promotes(tokens):
    """Quantised activations and the hand-over counts of whole layers: one CTA, two, all of them (short units: no K cut)."""
    from moeflow_b200.fixed import FixedEPLayer

    cfg = MoEConfig(hidden_size=512, moe_intermediate_size=256, n_routed_experts=16, top_k=4)
    w13, w2 = make_weights(cfg, 0, dtype=torch.float32)
    stack = lambda ts: torch.stack([t.view(torch.uint8) for t in ts]).view(torch.float8_e4m3fn).cuda()  # noqa: E731
    first, second = [quant_block_fp8(t) for t in w13], [quant_block_fp8(t) for t in w2]
    x, bias = make_hidden(tokens, cfg, 3, device="cuda"), make_bias(cfg, 1, device="cuda")
    logits = make_logits(tokens, cfg, 4, dist="zipf", device="cuda")
    outs = []
    for n_sms in (None, 1, 2):
        layer = FixedEPLayer(cfg, 0, 1, None, None, capacity=64, backend="cuda", device="cuda", wait_ns=50_000_000,
                             gemm_kwargs={"block_m": 64} | ({} if n_sms is None else {"n_sms": n_sms}))
        layer.set_weights_fp8(stack([q for q, _ in first]), torch.stack([s for _, s in first]).cuda(),
                              stack([q for q, _ in second]), torch.stack([s for _, s in second]).cuda())
        outs += [layer.forward(x, logits, bias)[:tokens].clone() for _ in range(3)]
        assert layer.check_status()["code"] == 0 and layer.plan[1:3].tolist() == [1, 1]
    assert all(torch.equal(o, outs[0]) for o in outs)


@pytest.mark.parametrize("hidden,inter", [(1152, 128), (4096, 384)])
@pytest.mark.parametrize("n_sms", [1, 2, 5])
def test_quantised_activations_of_long_whole_units(hidden, inter, n_sms):
    """Units of 9 and 32 K blocks, narrow and wide ones, many per CTA: a group's warps meet once per epilogue and write the next
    maxima a unit (of the other group's, when narrow) later.  Bytes, scales and output against the stand-alone kernels."""
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.ops.fp8 import dequant_rows, down_proj_fp8, gate_up_swiglu_fp8, quant_rows_1x128
    from moeflow_b200.ops.grouped_gemm import plan_from_offsets

    tokens, counts = 64, ([1, 40, 16, 7], [33, 15, 2, 14], [20, 32, 3, 9])  # rows per expert of each slot
    cfg = MoEConfig(hidden_size=hidden, moe_intermediate_size=inter, n_routed_experts=12, top_k=3)
    gen = torch.Generator().manual_seed(hidden)
    ids = torch.stack([torch.repeat_interleave(torch.arange(4 * k, 4 * k + 4), torch.tensor(c)) for k, c in enumerate(counts)], 1)
    ids = ids.to(torch.int32).cuda()
    weights = torch.rand(tokens, 3, generator=gen).cuda()
    stack = lambda ts: torch.stack([t.view(torch.uint8) for t in ts]).view(torch.float8_e4m3fn).cuda()  # noqa: E731
    first = [quant_block_fp8(torch.randn(2 * inter, hidden, generator=gen) * (2.0 / hidden**0.5)) for _ in range(12)]
    second = [quant_block_fp8(torch.randn(hidden, inter, generator=gen) / inter**0.5) for _ in range(12)]
    pack = (stack([q for q, _ in first]), torch.stack([s for _, s in first]).cuda(),
            stack([q for q, _ in second]), torch.stack([s for _, s in second]).cuda())
    layer = FixedEPLayer(cfg, 0, 1, None, None, capacity=tokens, backend="cuda", device="cuda", wait_ns=50_000_000,
                         gemm_kwargs={"block_m": 64, "n_sms": n_sms})
    layer.set_weights_fp8(*pack)
    xs_ = [make_hidden(tokens, cfg, seed, device="cuda") for seed in (3, 4, 5)]
    for x in xs_ * 3:
        layer.forward_routed(x, weights, ids)
    assert layer.check_status()["code"] == 0 and layer.plan[1:3].tolist() == [1, 1]

    offsets, n = layer.offsets.tolist(), tokens * 3
    assert [b - a for a, b in zip(offsets, offsets[1:])] == [c for slot in counts for c in slot]
    tp = plan_from_offsets(offsets, 64, x.device)
    xq, xs = quant_rows_1x128(x)
    rows = layer.entry_row[:n].clone()
    act = gate_up_swiglu_fp8(xq, xs, *pack[:2], tp, row_index=rows, limit=cfg.swiglu_limit)
    aq, a_s = quant_rows_1x128(act.contiguous())
    f = layer._fp8
    assert torch.equal(f["aq"][:n], aq.view(torch.uint8)) and torch.equal(f["as"][:n], a_s)
    assert torch.equal(layer.y[:n], down_proj_fp8(aq, a_s, *pack[2:], tp, row_scale=layer.entry_w[:n].clone()))
    xf = dequant_rows(xq, xs)[rows.long()]
    for e, (lo, hi) in enumerate(zip(offsets[:-1], offsets[1:])):
        gate, up = (xf[lo:hi] @ dequant_block_fp8(pack[0][e], pack[1][e]).t()).chunk(2, dim=-1)
        ref = torch.nn.functional.silu(gate.clamp(max=cfg.swiglu_limit)) * up.clamp(-cfg.swiglu_limit, cfg.swiglu_limit)
        # one bf16 rounding of every element (2**-9) on sums whose fp32 error is far below it
        assert normwise_rel_err(act[lo:hi], ref) < 4 * 2.0**-8
