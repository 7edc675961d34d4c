"""Routed experts whose last kernel adds two more rows: the three tensors added by hand, bit for bit."""

import pytest
import torch
from conftest import SMALL_GPU, replace

from moeflow_b200.testing import make_bias, make_hidden, make_logits, make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("capacity,tokens,valid,hidden", [(1, 1, 1, 256), (8, 5, 5, 512), (64, 64, 37, 512), (300, 257, 257, 4096), (16, 0, 0, 256)])
def test_forward_add(capacity, tokens, valid, hidden):
    from moeflow_b200.fixed import FixedEPLayer

    cfg = replace(SMALL_GPU, hidden_size=hidden)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    layer = FixedEPLayer(cfg, 0, 1, w13, w2, capacity=capacity, backend="cuda")
    x, lg, bias = make_hidden(tokens, cfg, 1, device="cuda"), make_logits(tokens, cfg, 2, device="cuda"), make_bias(cfg, 3, device="cuda")
    num = torch.tensor(valid, dtype=torch.int32, device="cuda")
    first, second = (torch.randn(tokens, hidden, generator=torch.Generator().manual_seed(s)).bfloat16().cuda() for s in (4, 5))
    guard = torch.full((tokens + 1, hidden), 7.0, dtype=torch.bfloat16, device="cuda")
    joined = []
    got = layer.forward_add(x, lg, bias, num, first, second, guard[:tokens], join=lambda: joined.append(1))
    assert joined == [1] and bool((guard[tokens] == 7).all())
    if tokens:
        routed = layer.forward(x, lg, bias, num)[:tokens]
        assert int(routed[valid:].count_nonzero()) == 0
        assert torch.equal(got, (first + routed) + second)
    assert layer.check_status()["code"] == 0


def test_what_it_refuses():
    from moeflow_b200.fixed import FixedEPLayer

    w13, w2 = make_weights(SMALL_GPU, 0, device="cuda")
    layer = FixedEPLayer(SMALL_GPU, 0, 1, w13, w2, capacity=8, backend="cuda")
    x, lg = make_hidden(4, SMALL_GPU, 1, device="cuda"), make_logits(4, SMALL_GPU, 2, device="cuda")
    ok = torch.zeros_like(x)
    for bad in (ok[:3], ok.float(), ok.cpu(), torch.zeros(4, 2 * x.shape[1], dtype=torch.bfloat16, device="cuda")[:, ::2]):
        with pytest.raises(ValueError):
            layer.forward_add(x, lg, None, None, bad, ok, ok)
    other = FixedEPLayer(SMALL_GPU, 0, 1, w13, w2, capacity=8, backend="cuda", gemm_kwargs={"fuse_return": True})
    with pytest.raises(ValueError):
        other.forward_add(x, lg, None, None, ok, ok, ok)


@pytest.mark.parametrize("tokens,valid,hidden", [(5, 3, 512), (257, 257, 4096)])
def test_the_output_may_be_one_of_the_summands(tokens, valid, hidden):
    """... and infinities and NaN in the summands are added like other values."""
    from moeflow_b200.fixed import FixedEPLayer

    cfg = replace(SMALL_GPU, hidden_size=hidden)
    w13, w2 = make_weights(cfg, 0, device="cuda")
    layer = FixedEPLayer(cfg, 0, 1, w13, w2, capacity=tokens, backend="cuda")
    x, lg, bias = make_hidden(tokens, cfg, 1, device="cuda"), make_logits(tokens, cfg, 2, device="cuda"), make_bias(cfg, 3, device="cuda")
    num = torch.tensor(valid, dtype=torch.int32, device="cuda")
    first, second = (torch.randn(tokens, hidden, generator=torch.Generator().manual_seed(s)).bfloat16().cuda() for s in (4, 5))
    first[0, 0], first[1, 9], second[1, 9], second[tokens - 1, hidden - 1] = float("inf"), float("inf"), float("-inf"), float("nan")
    want = (first + layer.forward(x, lg, bias, num)[:tokens]) + second
    assert bool(want[0, 0].isinf()) and bool(want[1, 9].isnan())
    for i in range(3):
        a, b = first.clone(), second.clone()
        out = (a, b, torch.empty_like(a))[i]
        assert layer.forward_add(x, lg, bias, num, a, b, out) is out
        torch.testing.assert_close(out, want, rtol=0, atol=0, equal_nan=True)
    assert layer.check_status()["code"] == 0
