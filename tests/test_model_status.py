"""A decode model answers for the status words of all its kernels (CPU: words are set by hand, nothing is launched)."""

from types import SimpleNamespace

import pytest
import torch

from moeflow_b200.models.glm_moe import DecodeModel
from moeflow_b200.ops import _lib


@pytest.mark.parametrize("part,layer", [(None, 0), ("routed", 0), ("router", 0), ("shared", 1)])
def test_a_wait_that_ran_out_anywhere_is_reported(part, layer):
    word = lambda: SimpleNamespace(status=torch.zeros(1, dtype=torch.int64))  # noqa: E731
    model = object.__new__(DecodeModel)
    model.routed = word()
    model.routed.check_status = lambda: _lib.decode_status(int(model.routed.status))
    model.layers = [{"router": word(), "shared": word()}, {"router": None, "shared": word()}, {"router": word(), "shared": SimpleNamespace()}]
    if part is not None:
        (model.routed if part == "routed" else model.layers[layer][part]).status.fill_(0x80105)
    assert model.check_status() == _lib.decode_status(0x80105 if part else 0)
