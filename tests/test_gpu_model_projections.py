"""The decode model's output projection, and the position that moves on next to the last experts."""

import pytest
import torch

from moeflow_b200 import MoEConfig

pytestmark = pytest.mark.gpu

CFG = MoEConfig(hidden_size=512, moe_intermediate_size=256, n_routed_experts=16, n_shared_experts=1, top_k=4)


@pytest.mark.parametrize("change", ["none", "other storage", "transposed, in place", "off the 16-byte grid"])
@pytest.mark.parametrize("batch", [1, 5, 16])
def test_output_projection_is_the_library_product_with_the_present_weights(batch, change):
    """Nothing of the weights is kept between steps, whatever happens to them in between."""
    from moeflow_b200.models.glm_moe import Attention, AttentionConfig

    attn = Attention(512, AttentionConfig(n_heads=8, n_kv_heads=2, head_dim=64, max_seq=24), batch, "cuda", 3)
    gen = torch.Generator().manual_seed(batch)
    x = torch.randn(batch, 512, generator=gen).bfloat16().cuda()
    pos = torch.tensor(9, device="cuda")
    mask = torch.full((1, 1, 1, 24), float("-inf"), dtype=torch.bfloat16, device="cuda")
    mask[..., :10] = 0
    attn.fill_cache(9, 5)
    wo = attn.wo
    attn.wo = torch.eye(512, dtype=torch.bfloat16, device="cuda")
    o = attn.delta(x, pos, mask)  # sums of one product and zeros: the attention itself
    attn.wo = wo.t().contiguous().t() if change.startswith("transposed") else wo
    first, kept = attn.delta(x, pos, mask), wo.data  # (the first storage stays allocated)
    if change == "other storage":
        wo.data = torch.randn(512, 512, generator=gen).bfloat16().cuda()
    elif change == "transposed, in place":
        attn.wo.mul_(-0.5)
    elif change == "off the 16-byte grid":
        attn.wo = torch.empty(512 * 512 + 1, dtype=torch.bfloat16, device="cuda")[1:].view(512, 512).copy_(wo)
    got = attn.delta(x, pos, mask)
    assert torch.equal(got, o @ attn.wo.t())
    assert kept is not None and (change != "none" or torch.equal(got, first))


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
        assert model.check_status()["code"] == 0
        runs.append(outs)
        model.close()
    assert all(torch.equal(a, b) for a, b in zip(*runs))
