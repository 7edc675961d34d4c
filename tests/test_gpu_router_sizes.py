"""Router kernel at the edges of its register batches (32 experts each, 16 of them), with ties and scores that vanish."""

import pytest
import torch

from moeflow_b200 import MoEConfig
from moeflow_b200.router import route

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("with_bias", [False, True])
@pytest.mark.parametrize("experts,top_k", [(4, 4), (31, 4), (32, 8), (33, 8), (100, 5), (288, 8), (511, 8), (512, 32), (513, 8)])
def test_router_kernel_at_the_edges_of_its_batches(experts, top_k, with_bias):
    from moeflow_b200.ops.kernels import router_topk

    cfg = MoEConfig(n_routed_experts=experts, top_k=top_k)
    gen = torch.Generator().manual_seed(experts)
    logits = torch.randn(9, experts, generator=gen)
    logits[1] = 0.25                                  # all tie: lowest ids, in order
    logits[2] = torch.randint(0, 3, (experts,), generator=gen).float()
    logits[3] = float("-inf")                         # scores of 0 everywhere
    logits[4, : experts // 2] = float("-inf")
    logits[5] = 200.0                                 # scores of 1 everywhere
    bias = 0.05 * torch.randn(experts, generator=gen) if with_bias else None
    w, ids = router_topk(logits.cuda(), None if bias is None else bias.cuda(), cfg)
    ref_w, ref_ids = route(logits, bias, cfg)
    assert torch.equal(ids.cpu().long(), ref_ids.long())
    torch.testing.assert_close(w.cpu(), ref_w, rtol=2e-6, atol=1e-7)  # a few fp32 roundings of the same expression
