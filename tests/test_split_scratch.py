"""Which scratch the argument blocks of a layer point at (CPU: the layer is built on host buffers and never launched)."""

import ctypes
import shutil

import pytest
import torch

from moeflow_b200 import MoEConfig


class _HostRegion:
    """A peer region of one rank in host memory."""

    world = 1

    def __init__(self, nbytes):
        self._bytes = torch.zeros(nbytes, dtype=torch.uint8)
        self.local = self
        self.nbytes = nbytes

    def view(self, offset, shape, dtype):
        n = torch.Size(shape).numel() * torch.empty(0, dtype=dtype).element_size()
        return self._bytes[offset : offset + n].view(dtype).view(shape)

    def table(self, offset):
        return torch.tensor([self._bytes.data_ptr() + offset])


@pytest.fixture
def host_layer(monkeypatch):
    from moeflow_b200 import fixed
    from moeflow_b200.ops import _lib, kernels

    if not _lib.LIB_PATH.exists() and shutil.which("nvcc") is None:
        pytest.skip("native library not built and no nvcc")
    monkeypatch.setattr(_lib, "available", lambda: True)
    for name in ("make_tile_tmap", "make_weight_tmap"):
        monkeypatch.setattr(kernels, name, lambda *a: ctypes.create_string_buffer(128))
    monkeypatch.setattr(kernels, "sm_count", lambda index: 148)

    def build(block_m, hidden=512, inter=256, **gemm_kwargs):
        cfg = MoEConfig(hidden_size=hidden, moe_intermediate_size=inter, n_routed_experts=4, top_k=2)
        region = _HostRegion(fixed.FixedEPLayer.peer_bytes(cfg, 1, 8))
        return fixed.FixedEPLayer(cfg, 0, 1, None, None, capacity=8, device="cpu", backend="cuda", peer_region=region,
                                  gemm_kwargs={"block_m": block_m, **gemm_kwargs})

    return build


@pytest.mark.parametrize("block_m", [32, 64, 128])
@pytest.mark.parametrize("handover", [True, False])
def test_the_two_gemms_of_a_layer_share_no_split_scratch(host_layer, block_m, handover):
    """With tile-level hand-over the down GEMM parks partial sums while gate/up units still wait for theirs.  Two token tiles
    of hidden 4096, intermediate 1536 on 148 SMs are cut into 48 gate/up and 64 down slots each, of the same size: in one
    scratch, the first tile's down sums lie on the second tile's gate/up sums."""
    layer = host_layer(block_m, tile_handover=handover)
    f = layer._fp8_buffers()
    lo, hi = layer._partial.data_ptr(), layer._partial.data_ptr() + 4 * layer._partial.numel()
    for first, second in ((layer._a_gemm1, layer._a_gemm2), (f["a1"], f["a2"])):
        spans = sorted((g.partial, g.partial + 4 * g.partial_floats) for g in (first, second))
        assert lo <= spans[0][0] < spans[0][1] <= spans[1][0] < spans[1][1] <= hi
        assert first.counters != second.counters and first.sched != second.sched
        assert all(g.partial % 16 == 0 and g.partial_floats == layer._a_meta.partial_floats for g in (first, second))
