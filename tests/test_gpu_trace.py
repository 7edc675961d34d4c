"""The stamps of ``cli/trace_layer.py``: every kernel that a forward launches leaves its own, in order."""

import pytest
import torch

from conftest import SMALL_GPU
from moeflow_b200.testing import make_hidden, make_logits, make_weights

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kwargs,launched", [({}, ("dispatch", "metadata", "reduce+push")),
                                             ({"meta_ctas": 1}, ("dispatch", "metadata", "reduce+push")),
                                             ({"fuse_return": True}, ("dispatch", "metadata", "combine"))])
def test_every_launched_kernel_is_stamped(kwargs, launched):
    from moeflow_b200.cli.trace_layer import SMALL_EVENTS, attach_traces
    from moeflow_b200.fixed import FixedEPLayer

    layer = FixedEPLayer(SMALL_GPU, 0, 1, *make_weights(SMALL_GPU, 0, device="cuda"), capacity=4, backend="cuda",
                         gemm_kwargs=kwargs, wait_ns=50_000_000)
    traces = attach_traces(layer)
    layer.forward(make_hidden(4, SMALL_GPU, 1, device="cuda"), make_logits(4, SMALL_GPU, 2, device="cuda"), None)
    assert layer.check_status()["code"] == 0
    at = {name: {ev: int(t) for ev, t in zip(SMALL_EVENTS[name], traces[name].tolist()) if t} for name in SMALL_EVENTS}
    assert [name for name in SMALL_EVENTS if at[name]] == list(launched)
    meta = at["metadata"]
    order = [meta[ev] for ev in ("loads issued", "warp 0 histogram", "histogram", "plan written", "entries placed")]
    assert order == sorted(order)
    assert at["dispatch"]["rows stored"] <= meta["loads issued"] and traces["gate/up GEMM"].any() and traces["down GEMM"].any()
    tail = at[launched[-1]]
    done = tail["row stored"] if "row stored" in tail else tail["row written"]
    assert meta["entries placed"] < done and int(traces["down GEMM"].max()) > meta["plan written"]
