"""The cut-cell volume pass on level sets near FP32's largest numbers, where the
products of its FP32 root search leave their range: per-cell volumes bit-exact
against the oracle."""
import numpy as np
import pytest

import oracle
from paritylib import make_gpu
from test_gpu_volume_columns import ball_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [112, 118, 121, 123, 125, 126, 130])
def test_large_levels(power):
    case = ball_case(3)
    case.levels[0].phi = case.levels[0].phi * 2.0 ** power
    orc = oracle.Oracle(case)
    gpu = make_gpu(case, "fp64")
    try:
        ref = orc.volume_mass(0)
        got = gpu.volume_mass(0, cells=True)
    finally:
        gpu.close()
    assert (ref["vol"] > 0).any()
    assert np.array_equal(got["vol"].ravel(), ref["vol"])
