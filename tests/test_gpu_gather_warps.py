"""256-row token tiles whose rows four extra warps gather, against the copy into expert-major order: same operands, same MMAs,
so the same bits, at the edges of the 16-row passes, of a wide tile and of a cut unit."""

import pytest
import torch
from conftest import SMALL_GPU, replace

from moeflow_b200.testing import make_bias, make_hidden, make_logits, make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("world,capacity,tokens,experts,top_k,hidden", [
    (1, 1, 1, 8, 2, 256), (1, 17, 15, 2, 1, 2048), (2, 40, 37, 4, 2, 256), (1, 257, 257, 1, 1, 512), (1, 700, 613, 8, 4, 256)])
def test_gathered_rows_equal_copied_rows_bitwise(world, capacity, tokens, experts, top_k, hidden):
    from moeflow_b200.fixed import FixedEPLayer, simulate_fixed
    from moeflow_b200.parallel.peer import PeerGroup

    cfg = replace(SMALL_GPU, n_routed_experts=experts, top_k=top_k, hidden_size=hidden)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    bias = make_bias(cfg, 1, device="cuda")
    xs = [make_hidden(tokens - r, cfg, 2 + r, device="cuda") for r in range(world)]
    lgs = [make_logits(tokens - r, cfg, 4 + r, device="cuda") for r in range(world)]
    per, outs = experts // world, []
    for permute in (True, False):
        regions = PeerGroup.local(world, FixedEPLayer.peer_bytes(cfg, world, capacity))
        layers = [FixedEPLayer(cfg, r, world, w13[r * per : (r + 1) * per], w2[r * per : (r + 1) * per], capacity=capacity,
                               backend="cuda", peer_region=regions[r], wait_ns=50_000_000,
                               gemm_kwargs={"block_m": 256, "permute_rows": permute}) for r in range(world)]
        for _ in range(2):
            got = [o.clone() for o in simulate_fixed(layers, xs, lgs, bias)]
        assert all(ly.check_status()["code"] == 0 for ly in layers)
        outs.append(got)
    for a, b in zip(*outs):
        assert a.abs().sum() > 0 and torch.equal(a, b)
