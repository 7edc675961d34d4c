"""Grouped GEMMs of the bf16 kernels into rows that do not start on 16 bytes: the 2-byte stores give what the 16-byte ones give."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("block_m", [32, 64, 128, 256])
@pytest.mark.parametrize("two_blocks", [False, True])
def test_down_into_rows_off_the_grid(block_m, two_blocks):
    from moeflow_b200.ops import _lib
    from moeflow_b200.ops.grouped_gemm import down_proj, plan_from_offsets
    from moeflow_b200.ops.kernels import make_weight_tmap, sm_count

    g = torch.Generator().manual_seed(block_m)
    offsets, inter, hidden = [0, 17, 17, 50, 130], 128, 512
    act = torch.randn(offsets[-1], inter, generator=g).bfloat16().cuda()
    w2 = torch.randn(4, hidden, inter, generator=g).bfloat16().cuda()
    scale = torch.rand(offsets[-1], generator=g).cuda() + 0.5
    tp = plan_from_offsets(offsets, block_m, act.device)
    want = down_proj(act, w2, tp, row_scale=scale, two_blocks=two_blocks)
    pitch = hidden + 3
    out = torch.full((offsets[-1] + 1, pitch), 7.0, dtype=torch.bfloat16, device="cuda")
    status = torch.zeros(1, dtype=torch.int64, device="cuda")
    args = _lib.GemmArgs(b_base=act.data_ptr(), b_pitch=inter * 2, tile_e=tp.tile_e.data_ptr(), tile_s=tp.tile_s.data_ptr(), tile_n=tp.tile_n.data_ptr(),
                         plan=tp.plan.data_ptr(), split_word=_lib.PLAN_SPLIT2, m_blocks=hidden // (256 if two_blocks else 128),
                         two_blocks=int(two_blocks), k_blocks=inter // 64, rows_per_expert=hidden, up_row_offset=128 if two_blocks else 0,
                         out=out.data_ptr(), out_pitch=pitch, row_scale=scale.data_ptr(), status=status.data_ptr(), wait_ns=200_000_000,
                         max_tiles=tp.tile_e.numel())
    tmap = make_weight_tmap(w2)
    _lib.check(_lib.lib().mf_gemm_down(tmap, C.byref(args), block_m, sm_count(0), _lib.stream_ptr()), "down")
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert torch.equal(out[: offsets[-1], :hidden], want)
    assert bool((out[:, hidden:] == 7).all()) and bool((out[offsets[-1]] == 7).all())
