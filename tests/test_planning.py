"""Host-side planning rules: tile rows, metadata CTAs, and the K-split rule shared with the metadata kernels."""

import shutil

import pytest

from moeflow_b200.fixed import choose_block_m, choose_meta_ctas


def test_tile_rows_follow_the_expected_rows_per_expert_not_the_worst_case():
    assert choose_block_m(128, 8, 288) == 64     # EP=1 decode: 3.5 rows per expert
    assert choose_block_m(128, 8, 36) == 64      # EP=8, T=128: 28 rows per expert (worst case would be 227)
    assert choose_block_m(256, 8, 36) == 128     # 57 rows per expert: one tile per expert instead of two for some
    assert choose_block_m(512, 8, 72) == 128     # 57 rows
    assert choose_block_m(512, 8, 144) == 64     # 28 rows
    assert choose_block_m(2048, 8, 144) == 256   # EP=2 prefill: 114 rows per expert
    assert choose_block_m(8192, 8, 36) == 256    # EP=8 long prefill: 1820 rows per expert
    assert choose_block_m(1, 8, 1) == 64


def test_tile_rows_for_layers_that_will_hold_e4m3_experts():
    assert choose_block_m(256, 8, 36, fp8=True) == 64      # 57 rows
    assert choose_block_m(2048, 8, 144, fp8=True) == 128   # 114 rows: the e4m3 kernels, no expansion
    assert choose_block_m(8192, 8, 144, fp8=True) == 128   # 455 rows
    assert choose_block_m(8192, 8, 36, fp8=True) == 256    # 1820 rows: expanded to bf16 per forward


def test_metadata_ctas_by_size():
    assert choose_meta_ctas(8, 148) == 1
    assert choose_meta_ctas(2048, 148) == 1
    assert choose_meta_ctas(8192, 148) == 1       # EP=8, 128 tokens per rank, top-8: still the one-pass single CTA
    assert choose_meta_ctas(8193, 148) == 65
    assert choose_meta_ctas(16384, 148) == 128
    assert choose_meta_ctas(1 << 20, 148) == 148
    assert choose_meta_ctas(16384, 8) == 8


@pytest.fixture(scope="module")
def plan_split():
    from moeflow_b200.ops import _lib

    if not _lib.LIB_PATH.exists() and shutil.which("nvcc") is None:
        pytest.skip("native library not built and no nvcc")
    return _lib.lib().mf_plan_split


def test_wide_tiles_are_not_split_for_an_uneven_last_round(plan_split):
    # EP=8, T=128: 40 token tiles x 12 blocks = 480 units of 64-column tiles, just over three rounds of 148 CTAs;
    # splitting K in two there doubled the gate/up GEMM's time
    assert plan_split(480, 64, 148, 1024, 4, 64) == 1
    assert plan_split(432, 64, 148, 1024, 4, 64) == 1
    assert plan_split(40 * 32, 24, 148, 2048, 8, 64) == 1


def test_decode_sizes_split_k_to_fill_the_sms(plan_split):
    assert plan_split(8 * 12, 64, 148, 4096, 4, 16) >= 2      # T=1: 8 experts x 12 blocks on 148 SMs
    assert plan_split(1 * 12, 64, 148, 4096, 4, 16) == 8
    assert plan_split(0, 64, 148, 4096, 4, 16) == 1
    assert plan_split(8 * 12, 64, 148, 100, 4, 16) == 1        # not enough partial-sum slots for any split


@pytest.mark.parametrize("units", [1, 7, 96, 148, 149, 480, 2640])
@pytest.mark.parametrize("k_blocks", [24, 64, 6])
@pytest.mark.parametrize("cols", [16, 64, 128])
def test_split_always_divides_k_and_fits_the_slots(plan_split, units, k_blocks, cols):
    s = plan_split(units, k_blocks, 148, 1024, 4, cols)
    assert s in (1, 2, 4, 8) and k_blocks % s == 0 and (s == 1 or (k_blocks // s >= 2 and units * s <= 1024))


def test_k_splits_of_e4m3_layers_divide_their_128_wide_blocks(plan_split):
    """The e4m3 kernels refuse any other plan.  Where the plain rule's split divides them, it is the one taken."""
    from moeflow_b200.ops import _lib

    steps = _lib.lib().mf_plan_split_steps
    refused = 0
    for blocks in range(1, 33):  # K = 128 .. 4096
        for units in (1, 2, 3, 8, 12, 22, 32, 96, 148, 149, 300, 432, 1024):
            for overhead, cols in ((4, 16), (8, 16), (4, 64), (8, 128)):
                plain, got = plan_split(units, 2 * blocks, 148, 4096, overhead, cols), steps(units, 2 * blocks, 2, 148, 4096, overhead, cols)
                assert blocks % got == 0 and got <= plain
                if blocks % plain == 0:
                    assert got == plain
                refused += blocks % plain != 0
                assert steps(units, 2 * blocks, 1, 148, 4096, overhead, cols) == plain
    assert refused > 0  # hidden 384 with intermediate 128, hidden 2048 with 1408 or (one tile) 1536
    assert plan_split(3, 6, 148, 4096, 4, 16) == 2 and steps(3, 6, 2, 148, 4096, 4, 16) == 1


def test_paired_tiles_in_place_of_128_rows():
    from moeflow_b200.fixed import paired_block_m

    assert paired_block_m(256, 8, 36) == 256   # 57 rows per expert
    assert paired_block_m(512, 8, 72) == 256
    assert paired_block_m(40, 8, 8) == 64      # 40 rows on 8 experts: fewer pair units than pairs
    assert paired_block_m(64, 8, 8) == 256     # 64 rows
    assert paired_block_m(1, 8, 0) == 64


def test_paired_tiles_by_the_layer_s_size():
    from moeflow_b200.fixed import paired_block_m

    assert paired_block_m(200, 8, 36, 512, 256) == 256 and paired_block_m(72, 8, 8, 512, 256) == 256  # all units under way at once
    assert paired_block_m(150, 8, 16, 512, 1024) == 128   # a down GEMM of few units
    assert paired_block_m(75, 8, 8, 2048, 1536) == 128
    assert paired_block_m(450, 8, 48, 1024, 512) == 128   # one to three rounds of units
    assert paired_block_m(300, 8, 32, 512, 1024) == 128
    assert paired_block_m(180, 8, 32, 4096, 512) == 128
    assert paired_block_m(40, 8, 8, 512, 1024) == 64
    assert paired_block_m(240, 8, 32, 4096, 1536) == 256  # 2e8 weights per projection
    assert paired_block_m(540, 8, 72, 7168, 2048) == 256


def test_where_the_router_s_logits_come_with_the_normalisation():
    from moeflow_b200.models.glm_moe import RouterLogits

    def fits(hidden, experts, rows, shared, capacity=1 << 20):
        router = object.__new__(RouterLogits)
        router.H, router.E, router.C = hidden, experts, capacity
        return router.fits_norm(rows, shared)

    for shared in (False, True):
        assert fits(4096, 36, 64, shared) and not fits(4096, 36, 65, shared) and not fits(4096, 72, 33, shared)
        assert fits(8192, 36, 32, shared) and not fits(8192, 36, 33, shared) and fits(16384, 36, 16, shared)
        assert not fits(16448, 1, 1, shared) and not fits(4096, 36, 0, shared) and not fits(4096, 36, 9, shared, capacity=8)
    # shorter rows: the limit of hidden 4096, and two launches next to a shared expert
    assert fits(512, 36, 64, False) and not fits(512, 36, 65, False) and not fits(4032, 1, 1, True)
