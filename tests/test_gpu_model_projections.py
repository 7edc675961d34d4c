"""The decode model's output projection on the dense kernel, and the position that moves on next to the last experts."""

import pytest
import torch

from moeflow_b200 import MoEConfig
from moeflow_b200.tolerances import normwise_rel_err

pytestmark = pytest.mark.gpu

CFG = MoEConfig(hidden_size=512, moe_intermediate_size=256, n_routed_experts=16, n_shared_experts=1, top_k=4)


@pytest.mark.parametrize("batch", [1, 5, 15, 16])
def test_attention_matches_the_library_projection(batch):
    from moeflow_b200.models.glm_moe import Attention, AttentionConfig

    acfg = AttentionConfig(n_heads=8, n_kv_heads=2, head_dim=64, max_seq=24)
    attn = Attention(512, acfg, batch, "cuda", 3)
    x = torch.randn(batch, 512, generator=torch.Generator().manual_seed(batch)).bfloat16().cuda()
    pos = torch.tensor(9, device="cuda")
    mask = torch.full((1, 1, 1, 24), float("-inf"), dtype=torch.bfloat16, device="cuda")
    mask[..., :10] = 0
    attn.fill_cache(9, 5)
    got = attn.delta(x, pos, mask)
    assert (attn._o is not None) == (batch < 16)
    attn.OWN_OUTPUT_BELOW, attn.wo = 0, attn.wo.clone()  # other weights are looked at anew
    ref = attn.delta(x, pos, mask)
    assert attn._o is None
    # both round fp32 sums of the same products to bf16 (2**-9 each)
    assert normwise_rel_err(got, ref.float()) < 2.0**-8


@pytest.mark.parametrize("n_layers,batch", [(0, 2), (1, 4), (3, 2)])
def test_position_and_mask_of_captured_steps(n_layers, batch):
    from moeflow_b200.models.glm_moe import AttentionConfig, DecodeModel

    acfg = AttentionConfig(n_heads=8, n_kv_heads=2, head_dim=64, max_seq=64)
    runs = []
    for captured in (True, False):
        model = DecodeModel(CFG, 0, 1, batch, n_layers, "cuda", acfg, seed=2)
        gen = torch.Generator().manual_seed(1)
        model.prefill_standin(16)
        if captured:
            model.capture()
            model.prefill_standin(16)
        outs = []
        for step in range(6):
            model.x.copy_(torch.randn(batch, 512, generator=gen).bfloat16())
            outs.append(model.step().clone())
            assert int(model.pos) == 17 + step and int((model.mask == 0).sum()) == 18 + step
        runs.append(outs)
        model.close()
    assert all(torch.equal(a, b) for a, b in zip(*runs))
