"""CVP in boxes of very different sizes against the oracle bit for bit: from some
1e19 on, the squares of the box's lengths leave FP32's range.  (Between 2^64 and
2^68 the assignment's own FP32 squares do in part, and the oracle takes 1e20 for
an infinite distance.)"""
import numpy as np
import pytest

import oracle
from mrsph import SPHMeshGeneration, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("power", [0, 40, 50, 62, 80])
def test_cvp_scale(power):
    case = cases.star_shape(3, 4, 3000)
    s, p = 2.0 ** power, case.params
    for k in ("min_dl", "max_dl"):
        p[k] *= s
    for k in ("box_l", "box_r"):
        p[k] = [v * s for v in p[k]]
    for lv in case.levels:
        lv.phi = lv.phi * s
        lv.box_l, lv.dpkg = [v * s for v in lv.box_l], [v * s for v in lv.dpkg]
    rng = np.random.default_rng(8)
    lo, hi = np.array(p["box_l"]), np.array(p["box_r"])
    xyz = lo + rng.random((5000, 3)) * (hi - lo)
    vp = lo + rng.random((40, 3)) * (hi - lo)
    gpu = SPHMeshGeneration(case, precision="fp64")
    gv, gl, gm, gr = gpu.partition_points(xyz, vp, max_iter=4)
    gpu.close()
    ov, ol, om, orr = oracle.cvp(3, p["box_l"], p["box_r"], xyz, vp, max_iter=4)
    assert np.array_equal(gl, ol) and np.array_equal(gv, ov) and np.array_equal(gm, om)
    assert gr["error_max"] == orr["error_max"]
