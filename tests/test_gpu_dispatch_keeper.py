"""The dispatch launch of up to 16 token positions, whose last CTA routes all tokens for itself and builds the layout."""

import dataclasses

import pytest
import torch
import test_gpu_dispatch_local as local
from conftest import SMALL_GPU

from moeflow_b200.fixed import FixedEPLayer
from moeflow_b200.ops.kernels import router_topk
from moeflow_b200.testing import make_bias, make_hidden, make_logits, make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e4m3", [False, True])
@pytest.mark.parametrize("tokens,capacity,experts,top_k,extra", [
    (16, 16, 512, 8, {}),            # as many token positions as warps, as many experts as threads
    (11, 16, 36, 3, {}),             # a top-k that is no power of two
    (13, 15, 24, 6, local.GROUPED),
    (5, 9, 17, 5, local.SOFTMAX),
    (17, 17, 36, 8, {}),             # one token position more: the form without that CTA
])
def test_layout(tokens, capacity, experts, top_k, extra, e4m3):
    local.test_layout_of_the_combined_launch(tokens, capacity, experts, top_k, extra, e4m3)


@pytest.mark.parametrize("tokens,capacity", [(1, 1), (9, 16)])
def test_given_routing_and_padding_rows(tokens, capacity):
    """Ids and weights from the caller, some of them none of this layer's, and fewer live rows than tokens."""
    cfg = dataclasses.replace(SMALL_GPU, n_routed_experts=24, top_k=6)
    layers = [FixedEPLayer(cfg, 0, 1, *make_weights(cfg, 0, device="cuda"), capacity=capacity, backend="cuda", wait_ns=50_000_000,
                           gemm_kwargs=kw) for kw in ({}, {"meta_ctas": 1})]
    assert layers[0].fuse_meta and not layers[1].fuse_meta
    x = make_hidden(tokens, cfg, 3, device="cuda")
    weights, ids = router_topk(make_logits(tokens, cfg, 4, device="cuda"), make_bias(cfg, 1, device="cuda"), cfg)
    ids[:, 1] = -1
    for live in (tokens, tokens // 2):
        valid = torch.tensor(live, dtype=torch.int32, device="cuda")
        outs = [ly.forward_routed(x, weights, ids, valid).clone() for ly in layers]
        assert all(ly.check_status()["code"] == 0 for ly in layers)
        assert torch.equal(*outs) and torch.equal(layers[0].offsets, layers[1].offsets) and torch.equal(layers[0].plan, layers[1].plan)
        assert torch.equal(layers[0].hit, layers[1].hit) and int(layers[0].hit.sum()) == live
