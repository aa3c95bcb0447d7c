"""CVP at the edges of its kernels' tiles, against the FP64 oracle bit for bit:
one VP, VP counts either side of a warp and of an 8-lane group, many VPs (a
face table of several tiles), point counts either side of a 2048-point chunk,
coincident VPs (planes without a direction), and enough iterations to pass a
convergence test."""
import numpy as np
import pytest

import oracle
from mrsph import SPHMeshGeneration, cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def handles():
    hs = {2: SPHMeshGeneration(cases.disc_hole_2d(spacing=0.02, grid=64), precision="fp64"),
          3: SPHMeshGeneration(cases.torus_3d(dx_min=0.03, dx_max=0.09, fine_pkg=32, nlevels=2), precision="fp32")}
    yield hs
    for h in hs.values():
        h.close()


@pytest.mark.parametrize("dim,n,vps,iters,weighted,coincident", [
    (3, 1, 1, 2, False, False), (2, 2047, 2, 41, False, False), (3, 2049, 7, 81, True, False),
    (3, 5000, 31, 5, True, False), (2, 5000, 33, 5, False, False), (3, 20000, 300, 3, True, False),
    (2, 4096, 9, 6, False, True), (3, 30000, 1024, 1, False, False)])
def test_cvp_sizes(handles, dim, n, vps, iters, weighted, coincident):
    gpu = handles[dim]
    p = gpu.case.params
    rng = np.random.default_rng(dim * 1000 + vps)
    lo, hi = np.array(p["box_l"]), np.array(p["box_r"])
    xyz = lo + rng.random((n, 3)) * (hi - lo)
    vp = lo + rng.random((vps, 3)) * (hi - lo)
    if coincident:
        vp[5] = vp[2]
    mass = 0.5 + rng.random(n) if weighted else None
    gv, gl, gm, gr = gpu.partition_points(xyz, vp, mass=mass, max_iter=iters)
    ov, ol, om, orr = oracle.cvp(dim, p["box_l"], p["box_r"], xyz, vp, mass=mass, max_iter=iters)
    assert np.array_equal(gl, ol)
    assert np.array_equal(gv, ov, equal_nan=True)
    assert np.array_equal(gm, om)
    assert (gr["iterations"], gr["converged"]) == (orr["iterations"], orr["converged"])
    assert np.array_equal([gr["error_max"], gr["total_energy"]], [orr["error_max"], orr["total_energy"]], equal_nan=True)
