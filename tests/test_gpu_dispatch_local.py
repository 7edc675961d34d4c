"""The dispatch launch of one rank that also builds the metadata: everything it leaves against the torch layout of the
same received rows and, bit for bit, against the two separate launches."""

import dataclasses

import pytest
import torch

from conftest import SMALL_GPU
from moeflow_b200.fixed import FixedEPLayer
from moeflow_b200.testing import make_bias, make_hidden, make_logits, make_weights
from moeflow_b200.weights import quant_block_fp8

pytestmark = pytest.mark.gpu

GROUPED = dict(n_group=4, topk_group=2)
SOFTMAX = dict(scoring_func="softmax", norm_topk_prob=False, routed_scaling_factor=1.0)


def _e4m3(w13, w2):
    packs = []
    for w in (w13, w2):
        qs, ss = zip(*(quant_block_fp8(w[e].float()) for e in range(w.shape[0])))
        packs += [torch.stack([q.view(torch.uint8) for q in qs]).view(torch.float8_e4m3fn), torch.stack(ss)]
    return packs


@pytest.mark.parametrize("e4m3", [False, True])
@pytest.mark.parametrize("tokens,capacity,experts,top_k,extra", [
    (1, 1, 8, 2, {}),                # one row, one warp of slot words
    (512, 512, 32, 8, {}),           # 4096 slot words exactly
    (500, 512, 8, 8, {}),            # every expert hit by every row
    (37, 64, 512, 8, {}),            # as many experts as threads
    (1365, 1365, 36, 3, {}),         # 4095 words, a top-k that is no power of two
    (100, 128, 24, 6, GROUPED),
    (33, 40, 17, 5, SOFTMAX),
    (0, 16, 8, 2, {}),
])
def test_layout_of_the_combined_launch(tokens, capacity, experts, top_k, extra, e4m3):
    cfg = dataclasses.replace(SMALL_GPU, n_routed_experts=experts, top_k=top_k, **extra)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    packs = _e4m3(w13, w2) if e4m3 else None

    def layer(**kwargs):
        if not e4m3:
            return FixedEPLayer(cfg, 0, 1, w13, w2, capacity=capacity, backend="cuda", wait_ns=50_000_000, gemm_kwargs=kwargs)
        ly = FixedEPLayer(cfg, 0, 1, None, None, capacity=capacity, backend="cuda", device="cuda", wait_ns=50_000_000,
                          gemm_kwargs={"block_m": 64, **kwargs})
        ly.set_weights_fp8(*packs)
        return ly

    one, two = layer(), layer(meta_ctas=1)
    assert one.fuse_meta and not two.fuse_meta
    bias = make_bias(cfg, 1, device="cuda")
    for seed, valid in ((3, None), (4, tokens // 2), (5, None)):  # buffers of the forward before are still full
        x, lg = make_hidden(tokens, cfg, seed, device="cuda"), make_logits(tokens, cfg, seed + 9, device="cuda")
        nv = None if valid is None else torch.tensor(valid, dtype=torch.int32, device="cuda")
        for ly in (one, two):
            ly.forward(x, lg, bias, nv, stop_after="META")
            assert ly.check_status()["code"] == 0
        _, local, wts = one.received_routing()
        live = tokens if valid is None else valid
        assert int((local >= 0).sum()) == live * top_k
        order, offsets, inv, entry_row, entry_slot = one._torch_layout(local)
        n = int(offsets[-1])
        assert torch.equal(one.offsets.long(), offsets) and torch.equal(one.inv.view_as(inv).long(), inv)
        assert torch.equal(one.entry_row[:n].long(), entry_row[:n]) and torch.equal(one.entry_slot[:n].long(), entry_slot[:n])
        assert torch.equal(one.entry_w[:n], wts[entry_row[:n], entry_slot[:n]])
        assert torch.equal(one.row_hits.long(), (local >= 0).sum(dim=1))
        counts = (offsets[1:] - offsets[:-1]).tolist()
        tiles = [(e, int(offsets[e]) + s, min(one.block_m, c - s)) for e, c in enumerate(counts) for s in range(0, c, one.block_m)]
        nt = int(one.plan[0])
        assert list(zip(one.tile_e[:nt].tolist(), one.tile_s[:nt].tolist(), one.tile_n[:nt].tolist())) == tiles
        assert torch.equal(one.plan, two.plan) and torch.equal(one.hit, two.hit)
        rows = [ly._recv_store[0, :live].view(torch.int16) for ly in (one, two)]  # bits: ids and weights are no bf16 values
        assert torch.equal(*rows) and torch.equal(one._recv_store[0, :live, : cfg.hidden_size], x[:live])
        if e4m3:
            assert torch.equal(one._fp8["xq"][:live], two._fp8["xq"][:live]) and torch.equal(one._fp8["xs"][:live], two._fp8["xs"][:live])
        assert torch.equal(one.forward(x, lg, bias, nv), two.forward(x, lg, bias, nv))
    assert one.check_status()["code"] == 0
