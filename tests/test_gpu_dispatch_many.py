"""Dispatch at prefill sizes (a warp per token, four per CTA): every stored row against what the router says, at capacities
that do not fill the last CTA, with fewer tokens than positions and with padding behind num_valid."""

import pytest
import torch

from moeflow_b200 import MoEConfig
from moeflow_b200.testing import make_bias, make_hidden, make_logits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("routed", [False, True])
@pytest.mark.parametrize("world,capacity,tokens,valid,hidden,experts,top_k", [
    (1, 1024, 1024, None, 512, 12, 4), (2, 514, 500, None, 512, 12, 4), (1, 1027, 1027, 1000, 256, 36, 8), (2, 1025, 900, None, 4096, 12, 3),
    (3, 1026, 1026, 1, 384, 288, 8), (1, 1030, 1030, None, 6400, 600, 2)])
def test_rows_stored_at_prefill_sizes(routed, world, capacity, tokens, valid, hidden, experts, top_k):
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.ops.kernels import router_topk
    from moeflow_b200.parallel.peer import PeerGroup

    cfg = MoEConfig(hidden_size=hidden, moe_intermediate_size=128, n_routed_experts=experts, top_k=top_k)
    regions = PeerGroup.local(world, FixedEPLayer.peer_bytes(cfg, world, capacity))
    layers = [FixedEPLayer(cfg, r, world, None, None, capacity=capacity, backend="cuda", device="cuda", peer_region=regions[r],
                           wait_ns=50_000_000) for r in range(world)]
    per, bias = experts // world, make_bias(cfg, 1, device="cuda")
    n = None if valid is None else torch.tensor([valid], dtype=torch.int32, device="cuda")
    for s, ly in enumerate(layers):
        x, logits = make_hidden(tokens, cfg, 5 + s, device="cuda"), make_logits(tokens, cfg, 9 + s, device="cuda")
        weights, ids = router_topk(logits, bias, cfg)
        hit = ly.stage_dispatch_pack(x, weights, ids, n) if routed else ly.stage_pack(x, logits, bias, n)
        torch.cuda.synchronize()
        live = torch.arange(tokens, device="cuda") < (tokens if valid is None else valid)
        for d, owner in enumerate(layers):
            on = (ids // per == d) & live[:, None]
            meta = owner._meta_view(owner._recv_store)[s]
            assert torch.equal(meta[:tokens, :top_k], torch.where(on, ids - d * per, -1).int())
            assert torch.equal(meta[:tokens, top_k : 2 * top_k].contiguous().view(torch.float32), torch.where(on, weights, 0.0))
            present = on.any(dim=1)
            assert torch.equal(meta[:tokens, 2 * top_k], present.int()) and torch.equal(hit[:tokens, d].bool(), present)
            assert not meta[tokens:, 2 * top_k].any() and (meta[tokens:, :top_k] == -1).all() and not hit[tokens:, d].any()
            assert torch.equal(owner._recv_store[s, :tokens, :hidden][present], x[present])
        assert int(ly._epoch) == 1
    for owner in layers:
        assert owner._disp_flags.tolist() == [capacity] * world
