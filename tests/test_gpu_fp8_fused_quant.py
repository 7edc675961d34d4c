"""e4m3 layers: the quantisers inside the metadata launch (received rows) and inside the gate/up epilogue (activations)
against the stand-alone quantiser on the same values, byte for byte, at the edges of the token tiles."""

import pytest
import torch

from moeflow_b200 import MoEConfig
from moeflow_b200.testing import make_bias, make_hidden, make_logits
from moeflow_b200.weights import quant_block_fp8

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block_m", [32, 64, 128])
@pytest.mark.parametrize("tokens,capacity,experts,hidden,inter,top_k", [
    (1, 1, 8, 256, 128, 2), (16, 16, 2, 256, 256, 1), (33, 40, 2, 512, 128, 2), (64, 64, 1, 384, 640, 1),
    (97, 128, 3, 512, 256, 3), (5, 8, 16, 4096, 256, 8)])
def test_fused_quantisers_equal_the_stand_alone_one(block_m, tokens, capacity, experts, hidden, inter, top_k):
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.ops.fp8 import gate_up_swiglu_fp8, quant_rows_1x128
    from moeflow_b200.ops.grouped_gemm import plan_from_offsets

    cfg = MoEConfig(hidden_size=hidden, moe_intermediate_size=inter, n_routed_experts=experts, top_k=top_k)
    gen = torch.Generator().manual_seed(tokens)
    q13, s13, q2, s2 = [], [], [], []
    for _ in range(experts):
        a, b = quant_block_fp8(torch.randn(2 * inter, hidden, generator=gen) * (2.0 / hidden**0.5))
        c, d = quant_block_fp8(torch.randn(hidden, inter, generator=gen) / inter**0.5)
        q13.append(a.view(torch.uint8)), s13.append(b), q2.append(c.view(torch.uint8)), s2.append(d)
    q13, q2 = (torch.stack(t).view(torch.float8_e4m3fn).cuda() for t in (q13, q2))
    s13, s2 = torch.stack(s13).cuda(), torch.stack(s2).cuda()
    layer = FixedEPLayer(cfg, 0, 1, None, None, capacity=capacity, device="cuda", backend="cuda",
                         gemm_kwargs={"block_m": block_m}, wait_ns=50_000_000)
    layer.set_weights_fp8(q13, s13, q2, s2)
    x, logits = make_hidden(tokens, cfg, 3, device="cuda"), make_logits(tokens, cfg, 4, device="cuda")
    for _ in range(2):  # the second forward finds the first one's scales, counters and maxima in the buffers
        layer.forward(x, logits, make_bias(cfg, 5, device="cuda"), stop_after="GEMM1")
    torch.cuda.synchronize()
    assert layer.check_status()["code"] == 0
    f = layer._fp8
    assert f["in_meta"]
    xq, xs = quant_rows_1x128(x)
    assert torch.equal(f["xq"][:tokens], xq.view(torch.uint8)) and torch.equal(f["xs"][:tokens], xs)

    offsets = layer.offsets.tolist()
    n = offsets[-1]
    assert n == tokens * top_k
    tp = plan_from_offsets(offsets, block_m, x.device)
    act = gate_up_swiglu_fp8(xq, xs, q13, s13, tp, row_index=layer.entry_row[:n].clone(), limit=cfg.swiglu_limit)
    aq, a_s = quant_rows_1x128(act.contiguous())
    if int(layer.plan[1]) == 1:  # uncut units add up in the same order, so the bytes agree
        assert torch.equal(f["aq"][:n], aq.view(torch.uint8)) and torch.equal(f["as"][:n], a_s)
    else:  # a K cut moves the last bit of some sums: scales within one bf16 step, codes within one e4m3 step
        torch.testing.assert_close(f["as"][:n], a_s, rtol=2.0**-7, atol=0)
        got = f["aq"][:n].view(torch.float8_e4m3fn).float().view(n, -1, 128) * f["as"][:n, :, None]
        want = aq.float().view(n, -1, 128) * a_s[:, :, None]
        step = want.abs() * 2.0**-3 + a_s[:, :, None] * 2.0**-8
        assert ((got - want).abs() <= step).all()
