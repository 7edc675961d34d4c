"""256-row tiles on CTA pairs against the same layer on one CTA (which takes the single form): the same products in the same
order, so the same bits, at the edges of a tile's halves, for gathered and boxed rows, odd and even block counts."""

import pytest
import torch

from moeflow_b200 import MoEConfig
from moeflow_b200.testing import make_hidden, make_weights

pytestmark = pytest.mark.gpu


def _layer(cfg, w13, w2, tokens, n_sms=None, **kw):
    from moeflow_b200.fixed import FixedEPLayer

    layer = FixedEPLayer(cfg, 0, 1, w13, w2, capacity=tokens, backend="cuda", gemm_kwargs={"block_m": 256, **kw}, wait_ns=200_000_000)
    if n_sms is not None:
        layer.n_sms = n_sms  # CTAs of the GEMMs; the plan stays the one for the whole device
    return layer


@pytest.mark.parametrize("hidden,inter", [(512, 256), (768, 128), (1024, 512)])
@pytest.mark.parametrize("counts", [(1, 16, 17, 31), (32, 33, 127, 128), (129, 0, 255, 256), (257, 500, 3, 64)])
@pytest.mark.parametrize("kw", [{"permute_rows": False}, {"permute_rows": True}, {"permute_rows": False, "b_tma": False}])
def test_pairs_equal_single_ctas_bitwise(hidden, inter, counts, kw):
    cfg = MoEConfig(hidden_size=hidden, moe_intermediate_size=inter, n_routed_experts=4, top_k=1)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    t = sum(counts)
    x = make_hidden(t, cfg, 1, device="cuda")
    g = torch.Generator().manual_seed(2)
    ids = torch.repeat_interleave(torch.arange(4), torch.tensor(counts))[torch.randperm(t, generator=g)].int()[:, None].cuda()
    weights = torch.rand(t, 1, generator=g).cuda() + 0.5
    outs = []
    for n_sms in (1, 2, 5, None):  # (an odd number of CTAs leaves one out)
        layer = _layer(cfg, w13, w2, t, n_sms, **kw)
        for _ in range(2):
            outs.append(layer.forward_routed(x, weights, ids).clone())
            assert layer.check_status()["code"] == 0
    assert outs[0].abs().sum() > 0
    assert all(torch.equal(o, outs[0]) for o in outs[1:])


@pytest.mark.parametrize("split", [1, 2, 4, 0])
def test_cut_units_of_pairs(split):
    """K splits add the same segments in the same order as one CTA does; stream-K cuts elsewhere (fp32 sums)."""
    from moeflow_b200.ops.grouped_gemm import gate_up_swiglu, plan_from_offsets

    offsets = [0, 200, 205, 461]
    g = torch.Generator().manual_seed(3)
    w13 = (torch.randn(3, 1024, 1024, generator=g) / 16).bfloat16().cuda()
    x = torch.randn(offsets[-1], 1024, generator=g).bfloat16().cuda()
    got = []
    for grid in (1, 2, 148):
        status = torch.zeros(1, dtype=torch.int64, device="cuda")
        got.append(gate_up_swiglu(x, w13, plan_from_offsets(offsets, 256, x.device), split=split, status=status, wait_ns=200_000_000, grid=grid).clone())
        assert int(status.item()) == 0
    for o in got[1:]:
        # (stream-K: activations rounded to bf16 once, so 2**-8 of one where the sums straddle a rounding point)
        assert torch.equal(o, got[0]) if split else (o.float() - got[0].float()).norm() < 2.0**-9 * got[0].float().norm()


def test_a_tile_that_is_too_tall_is_reported_and_not_stored():
    from moeflow_b200.ops.grouped_gemm import gate_up_swiglu, plan_from_offsets

    g = torch.Generator().manual_seed(4)
    w13 = (torch.randn(2, 512, 512, generator=g) / 16).bfloat16().cuda()
    x = torch.randn(400, 512, generator=g).bfloat16().cuda()
    tp = plan_from_offsets([0, 100, 400], 256, x.device)
    tp.tile_n[1] = 300
    status = torch.zeros(1, dtype=torch.int64, device="cuda")
    out = gate_up_swiglu(x, w13, tp, status=status, wait_ns=200_000_000)
    torch.cuda.synchronize()
    assert int(status.item()) & 0xFF == 7  # bad argument
    assert out[:100].abs().sum() > 0 and int(out[100:356].count_nonzero()) == 0


@pytest.mark.parametrize("experts,tokens,inter,block_m", [(36, 200, 256, 256), (8, 40, 256, 64), (8, 72, 256, 256), (36, 200, 384, 128)])
def test_layers_of_36_to_80_rows(experts, tokens, inter, block_m):
    """Tile height by rule: the same output as 64-row tiles within the rounding of activations and result (2**-9 each)."""
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.testing import make_bias, make_logits

    cfg = MoEConfig(hidden_size=512, moe_intermediate_size=inter, n_routed_experts=experts, top_k=8)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    x, lg, bias = make_hidden(tokens, cfg, 1, device="cuda"), make_logits(tokens, cfg, 2, device="cuda"), make_bias(cfg, 3, device="cuda")
    outs = []
    for kw in ({}, {"block_m": 64}):
        layer = FixedEPLayer(cfg, 0, 1, w13, w2, capacity=tokens, backend="cuda", gemm_kwargs=kw, wait_ns=200_000_000)
        outs.append(layer.forward(x, lg, bias)[:tokens].double())
        assert layer.check_status()["code"] == 0 and layer.block_m == kw.get("block_m", block_m) and not layer.permute_rows
    assert (outs[0] - outs[1]).norm() < 2 * 2.0**-8 * outs[1].norm()


def test_units_of_pairs_cut_in_eight():
    """The largest K split, segments of two K blocks: both GEMMs, against one CTA."""
    from moeflow_b200.ops.grouped_gemm import down_proj, gate_up_swiglu, plan_from_offsets

    offsets = [0, 31, 287, 288]
    g = torch.Generator().manual_seed(8)
    w = (torch.randn(3, 1024, 1024, generator=g) / 16).bfloat16().cuda()
    x = torch.randn(offsets[-1], 1024, generator=g).bfloat16().cuda()
    scale = torch.rand(offsets[-1], generator=g).cuda() + 0.5
    for call in (lambda tp, **kw: gate_up_swiglu(x, w, tp, **kw),
                 lambda tp, **kw: down_proj(x, w, tp, row_scale=scale, b_tma=False, two_blocks=True, **kw)):
        got = []
        for grid in (1, 2, 148):
            status = torch.zeros(1, dtype=torch.int64, device="cuda")
            got.append(call(plan_from_offsets(offsets, 256, x.device), split=8, status=status, wait_ns=200_000_000, grid=grid).clone())
            assert int(status.item()) == 0
        assert got[0].abs().sum() > 0 and all(torch.equal(o, got[0]) for o in got[1:])


@pytest.mark.parametrize("hidden,inter", [(4096, 256), (4096, 1536), (512, 2048)])
def test_long_k_loops_on_pairs_equal_single_ctas_bitwise(hidden, inter):
    counts = (256, 131, 0, 17)
    cfg = MoEConfig(hidden_size=hidden, moe_intermediate_size=inter, n_routed_experts=4, top_k=1)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    t = sum(counts)
    x = make_hidden(t, cfg, 1, device="cuda")
    g = torch.Generator().manual_seed(2)
    ids = torch.repeat_interleave(torch.arange(4), torch.tensor(counts))[torch.randperm(t, generator=g)].int()[:, None].cuda()
    weights = torch.rand(t, 1, generator=g).cuda() + 0.5
    outs = []
    for n_sms in (1, 7, None):
        layer = _layer(cfg, w13, w2, t, n_sms, permute_rows=False)
        outs.append(layer.forward_routed(x, weights, ids).clone())
        assert layer.check_status()["code"] == 0
    assert outs[0].abs().sum() > 0 and all(torch.equal(o, outs[0]) for o in outs[1:])


@pytest.mark.parametrize("block_m", [32, 64, 128, 256])
@pytest.mark.parametrize("two_blocks", [False, True])
def test_infinities_and_nan_stay_where_they_belong(block_m, two_blocks):
    """Through the epilogue's transposition: a token's row and a weight row's column, nothing else."""
    from moeflow_b200.ops.grouped_gemm import down_proj, gate_up_swiglu, plan_from_offsets

    offsets, inter, hidden = [0, 40, 40, 300], 128, 512
    g = torch.Generator().manual_seed(block_m)
    act = torch.randn(offsets[-1], inter, generator=g).bfloat16().cuda()
    w2 = torch.randn(3, hidden, inter, generator=g).bfloat16().cuda()
    tp = plan_from_offsets(offsets, block_m, act.device)
    clean = down_proj(act, w2, tp, two_blocks=two_blocks, b_tma=False).clone()
    bad_rows = {3: float("inf"), 39: float("nan"), 40: float("-inf"), 201: float("inf"), 299: float("nan")}
    bad_cols = {0: (5, float("inf")), 2: (hidden - 3, float("nan"))}  # expert: (weight row, value)
    act_bad, w_bad = act.clone(), w2.clone()
    for row, value in bad_rows.items():
        act_bad[row, row % inter] = value
    for e, (row, value) in bad_cols.items():
        w_bad[e, row, 7] = value
    y = down_proj(act_bad, w_bad, tp, two_blocks=two_blocks, b_tma=False)
    want, hit = clean.float(), torch.zeros_like(clean, dtype=torch.bool)
    for e, (lo, hi) in enumerate(zip(offsets, offsets[1:])):
        for row in [r for r in bad_rows if lo <= r < hi]:
            hit[row] = True
            want[row] = (act_bad[row].float() * w_bad[e].float()).sum(1)  # one value that is not finite decides every sum
        if e in bad_cols and hi > lo:
            col = bad_cols[e][0]
            hit[lo:hi, col] = True
            want[lo:hi, col] = (act_bad[lo:hi].float() * w_bad[e, col].float()).sum(1)
    assert torch.equal(y[~hit], clean[~hit])
    assert torch.equal(torch.isnan(y[hit]), torch.isnan(want[hit])) and not torch.isfinite(want[hit]).any()
    inf = torch.isinf(want[hit])
    assert torch.equal(y[hit][inf].float(), want[hit][inf])
    # gate/up: the other rows keep their bits (what a row with such values becomes is up to the clamp)
    w13 = torch.randn(3, 2 * inter, hidden, generator=g).bfloat16().cuda()
    x = torch.randn(offsets[-1], hidden, generator=g).bfloat16().cuda()
    plain = gate_up_swiglu(x, w13, tp).clone()
    for row, value in bad_rows.items():
        x[row, row] = value
    rows = [r for r in range(offsets[-1]) if r not in bad_rows]
    assert torch.equal(gate_up_swiglu(x, w13, tp)[rows], plain[rows])
