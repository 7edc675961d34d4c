"""The K-split rule with the costs that the layers state (CPU: the rule is callable on the host)."""

import shutil

import pytest


@pytest.fixture(scope="module")
def split():
    from moeflow_b200.ops import _lib

    if not _lib.LIB_PATH.exists() and shutil.which("nvcc") is None:
        pytest.skip("native library not built and no nvcc")
    return _lib.lib().mf_plan_split_costs


def test_costlier_cuts_only_lead_to_fewer_of_them(split):
    for units in (1, 7, 40, 96, 128, 148, 149, 252, 600, 672, 1792):
        for k, k_step, overhead, cols in ((64, 1, 4, 16), (64, 2, 4, 16), (24, 2, 8, 32), (8, 1, 4, 16), (48, 2, 4, 128)):
            plain, costly = (split(units, k, k_step, 148, 4096, overhead, cols, kb) for kb in (1, 8))
            assert costly <= plain and k // k_step % costly == 0 and (k >= 16 or units < 4 or plain == 1)


def test_e4m3_decode_units_stay_whole_and_bf16_ones_are_cut(split):
    assert split(96, 64, 2, 148, 4096, 4, 16, 8) == 1     # one token, 8 experts x 12 blocks
    assert split(600, 64, 2, 148, 4096, 4, 16, 8) == 1    # 8 tokens, 50 experts: the plain rule cuts these in two
    assert split(600, 64, 2, 148, 4096, 4, 16, 1) == 2
    assert split(96, 64, 1, 148, 4096, 4, 16, 1) == 4     # the same in bf16: cut
    assert split(12, 64, 2, 148, 4096, 4, 16, 8) == 8     # one expert on 148 SMs
    assert split(40, 8, 1, 148, 4096, 4, 16, 1) == 1      # hidden 512
