"""The cut-cell volume pass where its FP32 signs cannot decide: level sets
scaled down to FP32's smallest numbers (every sub-cube column then goes to the
refined FP64 corners) and up to large ones, planes through lattice points and
a curved surface, per-cell volumes bit-exact against the oracle."""
import numpy as np
import pytest

import oracle
from mrsph import cases
from paritylib import make_gpu
from test_gpu_volume_mass import dyadic_case

pytestmark = pytest.mark.gpu


def ball_case(dim):
    p = cases.default_params(dim)
    p.update(min_dl=1 / 8, max_dl=1 / 8, cell_ratio=2.0, box_l=[0, 0, 0], box_r=[1, 1, 1 if dim == 3 else 0], seed=1)

    def sdf(X, Y, Z):
        return 0.3 - np.sqrt((X - 0.51) ** 2 + (Y - 0.47) ** 2 + ((Z - 0.53) ** 2 if dim == 3 else 0.0))
    lv = cases.make_level(sdf, dim, [0, 0, 0], [1 / 4, 1 / 4, 1 / 4 if dim == 3 else 1.0], [4, 4, 4 if dim == 3 else 1])
    return cases.Case("ball", p, [lv], 100, steps=1)


@pytest.mark.parametrize("make", [lambda: ball_case(3), lambda: ball_case(2), lambda: dyadic_case(3, "tilted")],
                         ids=["ball3", "ball2", "tilted3"])
@pytest.mark.parametrize("power", [-120, -100, -40, 0, 60])
def test_scaled_levels(make, power):
    case = make()
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
