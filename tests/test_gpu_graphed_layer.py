"""``GraphedMoELayer`` replays on the caller's own buffers: device tensors, pinned blocks, changing pointers and row
counts, and back to the static buffers.  Every call must give exactly what an eager forward gives."""

import pytest
import torch

from moeflow_b200 import MoEConfig
from moeflow_b200.testing import make_bias, make_hidden, make_logits, make_weights

pytestmark = pytest.mark.gpu

CFG = MoEConfig(hidden_size=512, moe_intermediate_size=256, n_routed_experts=16, top_k=4)


def _make(capacity):
    from moeflow_b200.fixed import FixedEPLayer
    from moeflow_b200.models.routed_moe import GraphedMoELayer

    w13, w2 = make_weights(CFG, 0, device="cuda")
    bias = make_bias(CFG, 1, device="cuda")
    eager = FixedEPLayer(CFG, 0, 1, w13, w2, capacity=capacity, backend="cuda", wait_ns=50_000_000)
    graphed = GraphedMoELayer(FixedEPLayer(CFG, 0, 1, w13, w2, capacity=capacity, backend="cuda", wait_ns=50_000_000), bias).capture()

    def reference(x, logits):
        return eager.forward(x, logits, bias)[: x.shape[0]].clone()

    return graphed, reference


def _inputs(tokens, seed):
    return make_hidden(tokens, CFG, seed, device="cuda"), make_logits(tokens, CFG, seed + 50, device="cuda")


@pytest.mark.parametrize("capacity", [1, 16, 130])
def test_device_tensors_and_static_buffers_alternate(capacity):
    graphed, reference = _make(capacity)
    sizes = sorted({1, (capacity + 1) // 2, capacity})
    for seed, t in enumerate(sizes + sizes[::-1]):
        x, lg = _inputs(t, seed)
        want = reference(x, lg)
        assert torch.equal(graphed(x, lg), want)
        into = torch.full((t, CFG.hidden_size), 7.0, dtype=torch.bfloat16, device="cuda")
        assert graphed(x, lg, into) is into and torch.equal(into, want)
        # strided rows, wider dtypes and rows off the 16-byte grid take the copying path
        strided = torch.cat([x, x], dim=1)[:, : CFG.hidden_size]
        off = torch.cat([x.new_zeros(1), x.flatten()])[1:].view_as(x)
        for other in (strided, x.float(), off):
            assert t == 1 or not graphed._readable(other, lg)
            assert torch.equal(graphed(other, lg), want)
        assert torch.equal(graphed(x, lg.double()), want) and torch.equal(graphed(x, torch.cat([lg, lg], dim=1)[:, : CFG.n_routed_experts]), want)
        pinned = torch.zeros(t, CFG.hidden_size, dtype=torch.bfloat16).pin_memory()
        graphed(x.cpu().pin_memory(), lg.cpu().pin_memory(), pinned)
        torch.cuda.synchronize()
        assert torch.equal(pinned, want.cpu())
        graphed.load(x, lg)
        assert torch.equal(graphed.replay()[:t], want) and not graphed.replay()[t:].any()
    assert graphed.layer.check_status()["code"] == 0
    with pytest.raises(ValueError):
        graphed(*_inputs(capacity + 1, 0))
    graphed.close()


@pytest.mark.parametrize("capacity", [1, 32, 300])
def test_pinned_blocks(capacity):
    """300 rows are above the direct limit and take the copy engine's way."""
    graphed, reference = _make(capacity)
    blocks = [graphed.new_pinned_inputs() for _ in range(2)]
    for seed, t in enumerate([capacity, 1, (capacity + 1) // 2, capacity]):
        x, lg = _inputs(t, seed)
        want = reference(x, lg).cpu()
        block = blocks[seed % 2]
        block.x[:t].copy_(x)
        block.logits[:t].copy_(lg)
        block.set_rows(t)
        out = torch.full((capacity, CFG.hidden_size), 7.0, dtype=torch.bfloat16).pin_memory()
        graphed.step(block, out)
        torch.cuda.synchronize()
        assert torch.equal(out[:t], want) and (out[t:] == 7.0).all()  # rows past the batch stay the caller's
        assert torch.equal(graphed.step(block).cpu(), want)
        plain = torch.zeros(t, CFG.hidden_size, dtype=torch.bfloat16)  # pageable memory: copied
        graphed.step(block, plain)
        torch.cuda.synchronize()
        assert torch.equal(plain, want)
    assert graphed.layer.check_status()["code"] == 0
    graphed.close()


def test_pinned_outputs_that_the_caller_drops():
    """A pinned output dropped while its replay is still queued is held until that is done: pinned memory allocated in the
    meantime is not the same."""
    graphed, reference = _make(16)
    block = graphed.new_pinned_inputs()
    x, lg = _inputs(16, 3)
    want = reference(x, lg).cpu()
    block.x.copy_(x)
    block.logits.copy_(lg)
    block.set_rows(16)
    for _ in range(5):
        torch.cuda.synchronize()
        torch.cuda._sleep(50_000_000)
        dropped = torch.zeros(16, CFG.hidden_size, dtype=torch.bfloat16).pin_memory()
        graphed.step(block, dropped)
        del dropped
        later = [torch.full((16, CFG.hidden_size), 7.0, dtype=torch.bfloat16).pin_memory() for _ in range(3)]
        kept = torch.zeros(16, CFG.hidden_size, dtype=torch.bfloat16).pin_memory()
        graphed.step(block, kept)
        torch.cuda.synchronize()
        assert torch.equal(kept, want) and all((t == 7.0).all() for t in later)
    graphed.close()
    assert not graphed._host_refs and graphed._host_out is None


def test_the_graph_keeps_to_the_static_buffers():
    """``.graph`` replayed by its holder after a call on the caller's buffers: static inputs in, ``.out`` out, and nothing is
    written to what that call was given."""
    graphed, reference = _make(16)
    graph = graphed.graph
    (x, lg), (x2, lg2) = _inputs(9, 1), _inputs(5, 2)
    into = torch.empty(9, CFG.hidden_size, dtype=torch.bfloat16, device="cuda")
    graphed(x, lg, into)
    into.fill_(7.0)
    graphed.load(x2, lg2)
    graph.replay()
    assert torch.equal(graphed.out[:5], reference(x2, lg2)) and (into == 7.0).all()
    assert torch.equal(graphed(x, lg), reference(x, lg))
    graph.replay()
    assert torch.equal(graphed.out[:5], reference(x2, lg2))
    graphed.capture()  # again: the earlier executable graph goes
    assert torch.equal(graphed(x, lg, into), reference(x, lg))
    graphed.close()


def test_calls_on_two_streams_follow_one_another():
    """Nothing but the launch order separates them: they share the layer's buffers."""
    graphed, reference = _make(64)
    streams = [torch.cuda.Stream() for _ in range(2)]
    cases = [_inputs(t, t) for t in (64, 7)]
    want = [reference(*c) for c in cases]
    graphed.load(*cases[1])
    torch.cuda.synchronize()
    for _ in range(20):
        outs = [torch.zeros_like(w) for w in want]
        torch.cuda.synchronize()
        for c, out, stream in zip(cases, outs, streams):
            with torch.cuda.stream(stream):
                graphed(*c, out)
        with torch.cuda.stream(streams[0]):
            last = graphed.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(out, w) for out, w in zip(outs, want)) and torch.equal(last[:7], want[1])
    assert graphed.layer.check_status()["code"] == 0
    graphed.close()


def test_refused_inside_another_capture():
    """A replay cannot be captured; the refusal leaves the layer as it was."""
    graphed, reference = _make(16)
    x, lg = _inputs(9, 1)
    block = graphed.new_pinned_inputs()
    block.set_rows(9)
    out = torch.zeros(9, CFG.hidden_size, dtype=torch.bfloat16, device="cuda")
    for call in (lambda: graphed(x, lg), lambda: graphed(x, lg, out), lambda: graphed.step(block, out), graphed.replay):
        with pytest.raises(RuntimeError, match="captur"):
            with torch.cuda.graph(torch.cuda.CUDAGraph()):
                call()
        assert torch.equal(graphed(x, lg, out), reference(x, lg))
    graphed.close()
