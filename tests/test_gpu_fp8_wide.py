"""The 128-row e4m3 kernels: tile edges, an odd number of weight blocks, cut units, scale rows off the 16-byte grid."""

import pytest
import torch

from moeflow_b200 import MoEConfig
from moeflow_b200.testing import make_bias, make_hidden, make_logits, make_weights
from moeflow_b200.tolerances import normwise_rel_err
from moeflow_b200.weights import dequant_block_fp8, quant_block_fp8

pytestmark = pytest.mark.gpu


def _swiglu(h, limit):
    gate, up = h.chunk(2, dim=-1)
    gate, up = gate.clamp(max=limit), up.clamp(-limit, limit)
    return torch.nn.functional.silu(gate) * up


@pytest.mark.parametrize("counts", [[1], [3, 4, 5], [31, 0, 33], [127, 129], [256, 2]])
@pytest.mark.parametrize("hidden,inter,split", [(256, 128, 1), (384, 128, 1), (640, 384, 1), (1024, 512, 2), (1024, 512, 4), (768, 384, 0)])
def test_128_row_tiles_match_the_dequantised_definition(counts, hidden, inter, split):
    from moeflow_b200.ops.fp8 import dequant_rows, down_proj_fp8, gate_up_swiglu_fp8, quant_rows_1x128
    from moeflow_b200.ops.grouped_gemm import plan_from_offsets

    gen = torch.Generator().manual_seed(hidden + sum(counts))
    q13, s13, q2, s2 = [], [], [], []
    for _ in counts:
        a, b = quant_block_fp8(torch.randn(2 * inter, hidden, generator=gen) * (2.0 / hidden**0.5))
        c, d = quant_block_fp8(torch.randn(hidden, inter, generator=gen) / inter**0.5)
        q13.append(a.view(torch.uint8)), s13.append(b), q2.append(c.view(torch.uint8)), s2.append(d)
    q13, q2 = (torch.stack(t).view(torch.float8_e4m3fn).cuda() for t in (q13, q2))
    s13, s2 = torch.stack(s13).cuda(), torch.stack(s2).cuda()
    n = sum(counts)
    offsets = [sum(counts[:i]) for i in range(len(counts) + 1)]
    x = torch.randn(n + 3, hidden, generator=gen).bfloat16().cuda()
    idx = torch.randint(0, n + 3, (n,), generator=gen).int().cuda()
    scale = (torch.rand(n, generator=gen) + 0.5).cuda()
    tp = plan_from_offsets(offsets, 128, x.device)
    status = torch.zeros(1, dtype=torch.int64, device="cuda")
    kw = dict(split=split, status=status, wait_ns=50_000_000)
    xq, xs = quant_rows_1x128(x)
    padded = torch.zeros(n + 3, xs.shape[1] + 1, device="cuda")
    padded[:, 1:] = xs
    act = gate_up_swiglu_fp8(xq, xs, q13, s13, tp, row_index=idx, limit=10.0, **kw)
    assert torch.equal(gate_up_swiglu_fp8(xq, padded[:, 1:], q13, s13, tp, row_index=idx, limit=10.0, **kw), act)
    in_order = gate_up_swiglu_fp8(xq[idx.long()], xs[idx.long()], q13, s13, tp, limit=10.0, **kw)
    assert torch.equal(in_order, act), "rows by index and contiguous rows differ"
    aq, a_s = quant_rows_1x128(act.contiguous())
    y = down_proj_fp8(aq, a_s, q2, s2, tp, row_scale=scale, **kw)
    y_gathered = down_proj_fp8(aq, a_s, q2, s2, tp, row_scale=scale, b_tma=False, **kw)
    assert int(status) == 0
    assert torch.equal(y, y_gathered), "token tiles by TMA and by the gather differ"
    x_dq, a_dq = dequant_rows(xq, xs)[idx.long()], dequant_rows(aq, a_s)
    for e, (lo, hi) in enumerate(zip(offsets[:-1], offsets[1:])):
        if hi > lo:
            # one bf16 rounding of every element (2**-9) on sums whose fp32 error is far below it
            ref = _swiglu(x_dq[lo:hi] @ dequant_block_fp8(q13[e], s13[e]).t(), 10.0)
            assert normwise_rel_err(act[lo:hi], ref) < 4 * 2.0**-8
            ref = (a_dq[lo:hi] @ dequant_block_fp8(q2[e], s2[e]).t()) * scale[lo:hi, None]
            assert normwise_rel_err(y[lo:hi], ref) < 4 * 2.0**-8


class _EditedCalls:
    """The native library with ``edit(args)`` run on the arguments of every grouped GEMM first."""

    def __init__(self, real, edit):
        self._real, self._edit = real, edit

    def __getattr__(self, name):
        fn = getattr(self._real, name)
        if not name.startswith("mf_gemm_"):
            return fn

        def call(tmap, args, *rest):
            self._edit(args._obj)
            return fn(tmap, args, *rest)

        return call


@pytest.fixture
def edit_calls(monkeypatch):
    from moeflow_b200.ops import _lib

    real = _lib.lib()
    return lambda edit: monkeypatch.setattr(_lib, "lib", lambda: _EditedCalls(real, edit))


def _down_problem(counts, hidden, inter, seed=0):
    """``(codes, scales, w2 codes, w2 scales, plan)`` of a down projection on 128-row tiles."""
    from moeflow_b200.ops.fp8 import quant_rows_1x128
    from moeflow_b200.ops.grouped_gemm import plan_from_offsets

    gen = torch.Generator().manual_seed(seed)
    packs = [quant_block_fp8(torch.randn(hidden, inter, generator=gen) / inter**0.5) for _ in counts]
    w2 = torch.stack([q.view(torch.uint8) for q, _ in packs]).view(torch.float8_e4m3fn).cuda()
    s2 = torch.stack([s for _, s in packs]).cuda()
    aq, a_s = quant_rows_1x128(torch.randn(sum(counts), inter, generator=gen).bfloat16().cuda())
    offsets = [sum(counts[:i]) for i in range(len(counts) + 1)]
    return aq, a_s, w2, s2, plan_from_offsets(offsets, 128, aq.device)


@pytest.mark.parametrize("split", [0, 1, 2])
@pytest.mark.parametrize("blocks", [1, 3, 4])
def test_only_the_weight_blocks_asked_for_are_computed(edit_calls, blocks, split):
    from moeflow_b200.ops.fp8 import down_proj_fp8

    aq, a_s, w2, s2, tp = _down_problem([5, 140], 640, 256)
    whole = down_proj_fp8(aq, a_s, w2, s2, tp, split=split)
    edit_calls(lambda a: setattr(a, "m_blocks", blocks))
    some = down_proj_fp8(aq, a_s, w2, s2, tp, split=split)
    assert some[:, blocks * 128 :].abs().sum() == 0
    if split:  # (stream-K cuts the shorter line of work elsewhere)
        assert torch.equal(some[:, : blocks * 128], whole[:, : blocks * 128])
    else:
        # a cut moves the last bit of an fp32 sum: some elements round to the other bf16 neighbour, 2**-8 of themselves
        assert normwise_rel_err(some[:, : blocks * 128], whole[:, : blocks * 128]) < 2.0**-8


@pytest.mark.parametrize("split", [0, 1, 2])
@pytest.mark.parametrize("counts", [[1], [7, 0, 20], [128, 129, 15]])
def test_rows_by_index_and_by_tensor_map_in_both_gemms(edit_calls, counts, split):
    """The down GEMM takes a row index and needs no tensor map; the gate/up GEMM reads a caller's map and not b_base."""
    from moeflow_b200.ops.fp8 import _gemm_fp8, down_proj_fp8, gate_up_swiglu_fp8

    n = sum(counts)
    aq, a_s, w2, s2, tp = _down_problem(counts, 512, 256)
    idx = torch.randperm(n, generator=torch.Generator().manual_seed(n)).int().cuda()
    status = torch.zeros(1, dtype=torch.int64, device="cuda")
    kw = dict(limit=None, split=split, status=status, wait_ns=50_000_000, grid=None)
    by_index = _gemm_fp8(False, aq, a_s, w2, s2, tp, torch.zeros(n, 512, dtype=torch.bfloat16, device="cuda"), idx, None, **kw)
    in_order = down_proj_fp8(aq[idx.long()], a_s[idx.long()], w2, s2, tp, split=split, status=status)
    assert int(status) == 0 and in_order.abs().sum() > 0 and torch.equal(by_index, in_order)

    gathered = gate_up_swiglu_fp8(aq, a_s, w2, s2, tp, limit=None, split=split, status=status)
    edit_calls(lambda a: setattr(a, "b_base", None))
    mapped = _gemm_fp8(True, aq, a_s, w2, s2, tp, torch.zeros(n, 256, dtype=torch.bfloat16, device="cuda"), None, None, b_tma=True, **kw)
    assert int(status) == 0 and gathered.abs().sum() > 0 and torch.equal(mapped, gathered)


@pytest.mark.parametrize("split,grid", [(0, 1), (0, 3), (0, 8), (0, 148), (2, 148), (4, 5)])
@pytest.mark.parametrize("hidden,shift", [(128, 0), (384, 0), (640, 0), (1024, 0), (384, 1), (384, 2)])
def test_cut_down_units_stay_inside_the_scratch_of_one_block_units(edit_calls, hidden, shift, split, grid):
    """A unit of two weight blocks needs no more scratch than two of one: as many accumulators of 128 x 128 sums as units of
    one block have segments (stream-K: two per CTA that has a K step).  ``shift``: floats from a 16-byte boundary."""
    from moeflow_b200.ops.fp8 import dequant_rows, down_proj_fp8

    aq, a_s, w2, s2, tp = _down_problem([30, 128, 131], hidden, 512)
    units = tp.n_tiles * (hidden // 128)
    accumulators = 2 * min(units * 4, grid) if split == 0 else units * split
    floats = accumulators * 128 * 128
    scratch = torch.full((shift + floats + 4096,), 77.0, device="cuda")[shift:]
    status = torch.zeros(1, dtype=torch.int64, device="cuda")
    checked = [floats]

    def shrink(a):
        a.partial, a.partial_floats = scratch.data_ptr(), checked[0]

    edit_calls(shrink)
    ref = dequant_rows(aq, a_s)
    ref = torch.cat([r @ dequant_block_fp8(w2[e], s2[e]).t() for e, r in enumerate(ref.split([30, 128, 131]))])
    for checked[0] in (floats, 0):  # 0: the kernel is not told how much there is
        y = down_proj_fp8(aq, a_s, w2, s2, tp, split=split, status=status, grid=grid, wait_ns=50_000_000)
        assert int(status) == 0 and (scratch[floats:] == 77).all()
        assert normwise_rel_err(y, ref) < 4 * 2.0**-8  # one bf16 rounding of sums whose fp32 error is far below it
    checked[0] = floats - 1  # refused on the device, nothing stored
    y = down_proj_fp8(aq, a_s, w2, s2, tp, split=split, status=status, grid=grid, wait_ns=50_000_000)
    assert int(status) != 0 and y.abs().sum() == 0


@pytest.mark.parametrize("block_m", [32, 64, 128])
@pytest.mark.parametrize("split", [1, 2])
def test_tiles_without_rows_are_passed_over(block_m, split):
    """In front of the first row and behind the last one: such a tile has no last row that could be read in place of one."""
    import dataclasses

    from moeflow_b200.ops import _lib
    from moeflow_b200.ops.fp8 import _gemm_fp8, down_proj_fp8
    from moeflow_b200.ops.grouped_gemm import plan_from_offsets

    aq, a_s, w2, s2, _ = _down_problem([5, 70], 512, 256)
    tp = plan_from_offsets([0, 5, 75], block_m, aq.device)
    i32 = dict(dtype=torch.int32, device="cuda")
    more = dataclasses.replace(
        tp, n_tiles=tp.n_tiles + 2, plan=tp.plan.clone(),
        **{k: torch.cat([torch.tensor([first], **i32), getattr(tp, k), torch.tensor([last], **i32)])
           for k, first, last in (("tile_e", 0, 1), ("tile_s", 0, 75), ("tile_n", 0, 0))})
    more.plan[_lib.PLAN_N_TILES] = more.n_tiles
    idx = torch.randperm(75, generator=torch.Generator().manual_seed(1)).int().cuda()
    status = torch.zeros(1, dtype=torch.int64, device="cuda")
    outs = []
    for plan in (tp, more):
        act = torch.zeros(75, 256, dtype=torch.bfloat16, device="cuda")
        _gemm_fp8(True, aq, a_s, w2, s2, plan, act, idx, None, None, split, status, 50_000_000, None)
        outs.append([act, *(down_proj_fp8(aq, a_s, w2, s2, plan, split=split, status=status, b_tma=b_tma) for b_tma in (True, False))])
    assert int(status) == 0
    for a, b in zip(*outs):
        assert a.abs().sum() > 0 and torch.equal(a, b)


@pytest.mark.parametrize("block_m,box_rows", [(32, 16), (32, 48), (64, 32), (64, 128)])
def test_box_rows_mean_nothing_to_tiles_of_up_to_64_rows(edit_calls, block_m, box_rows):
    """Their boxes hold a whole tile, whatever the field says."""
    from moeflow_b200.ops.fp8 import down_proj_fp8
    from moeflow_b200.ops.grouped_gemm import plan_from_offsets

    aq, a_s, w2, s2, _ = _down_problem([5, 70], 512, 256)
    tp = plan_from_offsets([0, 5, 75], block_m, aq.device)
    y = down_proj_fp8(aq, a_s, w2, s2, tp)
    edit_calls(lambda a: setattr(a, "b_box_rows", box_rows))
    assert y.abs().sum() > 0 and torch.equal(down_proj_fp8(aq, a_s, w2, s2, tp), y)


@pytest.mark.parametrize("rows,apart", [(5, 8 << 30), (34, 1 << 30)])
@pytest.mark.parametrize("block_m", [64, 128])
def test_gathered_rows_over_more_than_32_gib(block_m, rows, apart):
    """The last row lies 2**31 chunks of 16 bytes behind the first, or more."""
    from moeflow_b200.ops.fp8 import _gemm_fp8
    from moeflow_b200.ops.grouped_gemm import plan_from_offsets

    if torch.cuda.mem_get_info()[0] < 38 << 30:
        pytest.skip("needs 38 GiB of device memory")
    aq, a_s, w2, s2, _ = _down_problem([rows], 512, 256)
    tp = plan_from_offsets([0, rows], block_m, aq.device)
    far = torch.empty((rows - 1) * apart + 256, dtype=torch.uint8, device="cuda").as_strided((rows, 256), (apart, 1))
    far.copy_(aq.view(torch.uint8))
    far = far.view(torch.float8_e4m3fn)
    idx = torch.randperm(rows, generator=torch.Generator().manual_seed(2)).int().cuda()
    for gate_up, cols in ((True, 256), (False, 512)):
        near, away = (_gemm_fp8(gate_up, x, a_s, w2, s2, tp, torch.zeros(rows, cols, dtype=torch.bfloat16, device="cuda"), idx, None,
                                None, 1, None, 50_000_000, None) for x in (aq, far))
        assert near.abs().sum() > 0 and torch.equal(near, away)
    del far
    torch.cuda.empty_cache()


@pytest.mark.parametrize("tokens,hidden,inter", [(1, 384, 256), (50, 640, 384), (300, 512, 256)])
def test_layer_on_128_row_tiles_matches_64_row_tiles(tokens, hidden, inter):
    """Whole layers: the plan counts pairs of weight blocks for the down GEMM, and every tile is handed over complete."""
    from moeflow_b200.fixed import FixedEPLayer

    cfg = MoEConfig(hidden_size=hidden, moe_intermediate_size=inter, n_routed_experts=4, top_k=2)
    w13, w2 = make_weights(cfg, 0, dtype=torch.float32)
    packs = [(*quant_block_fp8(w13[e]), *quant_block_fp8(w2[e])) for e in range(4)]
    weights = [torch.stack([p[i].view(torch.uint8) if i in (0, 2) else p[i] for p in packs]).cuda() for i in range(4)]
    weights = [w.view(torch.float8_e4m3fn) if w.dtype == torch.uint8 else w for w in weights]
    bias = make_bias(cfg, 1, device="cuda")
    x, logits = make_hidden(tokens, cfg, 2, device="cuda"), make_logits(tokens, cfg, 3, device="cuda")
    outs = []
    for block_m in (64, 128):
        layer = FixedEPLayer(cfg, 0, 1, None, None, capacity=tokens + 3, backend="cuda", device="cuda",
                             gemm_kwargs={"block_m": block_m}, wait_ns=50_000_000)
        layer.set_weights_fp8(*weights)
        for _ in range(2):
            out = layer.forward(x, logits, bias).clone()
        assert layer.check_status()["code"] == 0
        outs.append(out)
    # a K cut may move a bf16 activation by a step and with it the e4m3 code of some (2**-3 of the element): of 1 in 30
    # codes at most, 2**-3 / sqrt(30) = 0.023 of the norm
    assert normwise_rel_err(outs[1], outs[0]) < 0.023
    # bound to bf16 experts afterwards, the layer's plan is that of the bf16 kernels again
    layer.set_weights(torch.stack([dequant_block_fp8(p[0], p[1]) for p in packs]).bfloat16().cuda(),
                      torch.stack([dequant_block_fp8(p[2], p[3]) for p in packs]).bfloat16().cuda())
    out = layer.forward(x, logits, bias)
    assert layer.check_status()["code"] == 0
    assert normwise_rel_err(out, outs[0]) < 0.06  # e4m3 activations against bf16 ones


def _packed(cfg, device="cuda"):
    """e4m3 expert weights of a layer: ``(w13, scales, w2, scales)``."""
    w13, w2 = make_weights(cfg, 0, dtype=torch.float32, device=device)
    packs = [[*quant_block_fp8(a), *quant_block_fp8(b)] for a, b in zip(w13, w2)]
    codes = lambda i: torch.stack([p[i].view(torch.uint8) for p in packs]).view(torch.float8_e4m3fn)  # noqa: E731
    return codes(0), torch.stack([p[1] for p in packs]), codes(2), torch.stack([p[3] for p in packs])


@pytest.mark.parametrize("hidden,inter,experts,tokens,top_k,both", [
    (4096, 1536, 2, 9, 1, True), (4096, 1536, 4, 24, 2, True), (4096, 1536, 1, 40, 1, True), (640, 1536, 3, 50, 1, False),
    (384, 2048, 2, 5, 1, False)])
def test_layers_with_cut_down_units(hidden, inter, experts, tokens, top_k, both):
    """Cut units in both GEMMs, or in the down GEMM with a last unit of one block.  With tile-level hand-over down units run
    next to gate/up units whose partial sums still lie in scratch: the bits are those without it, in every forward."""
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.ops import _lib

    cfg = MoEConfig(hidden_size=hidden, moe_intermediate_size=inter, n_routed_experts=experts, top_k=top_k)
    weights = _packed(cfg)
    bias = make_bias(cfg, 1, device="cuda")
    inputs = [(make_hidden(tokens, cfg, s, device="cuda"), make_logits(tokens, cfg, 9 + s, device="cuda")) for s in (2, 3)]

    def layer(block_m, **kw):
        ly = FixedEPLayer(cfg, 0, 1, None, None, capacity=tokens, backend="cuda", device="cuda",
                          gemm_kwargs={"block_m": block_m, **kw}, wait_ns=50_000_000)
        ly.set_weights_fp8(*weights)
        return ly

    chained, apart, narrow = layer(128), layer(128, tile_handover=False), layer(64)
    want = [apart.forward(x, lg, bias).clone() for x, lg in inputs]
    for i in range(20):
        assert torch.equal(chained.forward(*inputs[i & 1], bias), want[i & 1])
        cuts = chained.plan[[_lib.PLAN_SPLIT1, _lib.PLAN_SPLIT2]].tolist()
        assert cuts[1] > 1 and (cuts[0] > 1 or not both)
    # as in the test above: a K cut may move the e4m3 code of 1 in 30 activations at most
    assert normwise_rel_err(narrow.forward(*inputs[0], bias), want[0]) < 0.023
    assert all(ly.check_status()["code"] == 0 for ly in (chained, apart, narrow))


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_infinities_and_nan_stay_in_their_own_row(bad):
    """The other rows' bits do not change, and the row's codes and scales are those of the 64-row kernel."""
    from moeflow_b200.fixed import FixedEPLayer

    cfg = MoEConfig(hidden_size=512, moe_intermediate_size=256, n_routed_experts=2, top_k=1)
    weights, bias = _packed(cfg), make_bias(cfg, 1, device="cuda")
    x, logits = make_hidden(150, cfg, 2, device="cuda"), make_logits(150, cfg, 3, device="cuda")
    outs = {}
    for block_m in (64, 128):
        layer = FixedEPLayer(cfg, 0, 1, None, None, capacity=150, backend="cuda", device="cuda",
                             gemm_kwargs={"block_m": block_m}, wait_ns=50_000_000)
        layer.set_weights_fp8(*weights)
        clean = layer.forward(x, logits, bias).clone()
        spoilt = x.clone()
        spoilt[70, 200] = bad
        out = layer.forward(spoilt, logits, bias).clone()
        assert layer.check_status()["code"] == 0
        rest = torch.arange(150, device="cuda") != 70
        assert torch.equal(out[rest], clean[rest])
        entry = int(layer.inv[70])
        outs[block_m] = [layer._fp8[k][entry].clone().view(torch.uint8) for k in ("aq", "as")]
    for a, b in zip(outs[64], outs[128]):
        assert torch.equal(a, b)
