"""The cost rule of the flux launches (csrc/device/flux_cut.hpp)."""
import pytest

from config_cases import FORM_GRIDS
from flux_cuts import FP64_GRIDS, MIXED_GRIDS, fp64_cut, march_cut


def test_the_grids_of_the_gpu_tests_take_every_cut():
    """... or test_gpu_tuning would compare less than it says."""
    assert {g: fp64_cut(g) for g in FP64_GRIDS} == FP64_GRIDS
    assert {g: [march_cut(v, g) for v in range(4)] for g in MIXED_GRIDS} == MIXED_GRIDS
    assert set(FP64_GRIDS.values()) == {"rows", 1, 2, 4, 8}
    for q in range(2):  # y, z
        assert {m[q] for cuts in MIXED_GRIDS.values() for m in cuts} == {1, 2, 4, 8, 16}
    assert [fp64_cut((n, n // 2, 1), air=True) for n in (48, 256)] == ["rows", 1]
    # every model: rows in 3-D for air, rows and columns of three lengths for mixtures, both in 2-D
    assert [fp64_cut(g) for g in FORM_GRIDS] == ["rows", 1, 2, 8, "rows", 1]
    assert [fp64_cut(g, air=True) for g in FORM_GRIDS] == ["rows"] * 5 + [1]


def test_the_workloads_take_the_cuts_they_were_measured_with():
    assert fp64_cut((24, 16, 8)) == "rows" and fp64_cut((160, 96, 64)) == 4 and fp64_cut((384, 192, 64)) == 8
    assert fp64_cut((128, 64, 1), air=True) == "rows"
    assert march_cut(0, (24, 16, 8)) == (1, 1) and march_cut(0, (96, 64, 32)) == (2, 2)
    assert march_cut(0, (384, 192, 64)) == (8, 8) and march_cut(1, (512, 256, 224)) == (16, 16)


@pytest.mark.parametrize("sms", [1, 74, 148, 296])
def test_blocks_count_together(sms):
    half, whole = (96, 97, 61), (192, 97, 61)
    assert fp64_cut(half, half, sms=sms) == fp64_cut(whole, sms=sms)
    assert march_cut(0, half, half, sms=sms) == march_cut(0, whole, sms=sms)


def test_few_sms_take_long_columns():
    assert fp64_cut((24, 16, 8), sms=1) == 8 and march_cut(0, (160, 96, 64), sms=1) == (8, 8)
