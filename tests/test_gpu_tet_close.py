"""Tetrahedra of particles far closer to one another than their balls are wide:
spacings whose sixth power, and then whose fourth, FP32 cannot hold, and
twins at a normal spacing.  Mesh and counters equal the oracle's on the same
particles and rows."""
import numpy as np
import pytest

import oracle
from mrsph import SPHMeshGeneration, cases
from test_gpu_mesh_paths import _lattice

pytestmark = pytest.mark.gpu


def _check(xyz):
    case = cases.torus_3d(dx_min=0.03, dx_max=0.09, fine_pkg=32, nlevels=2)
    gpu = SPHMeshGeneration(case, precision="fp64", neighbor_cap=2048)
    gpu.set_state({"xyz": xyz})
    gpu.run_phase(3)
    p = gpu.particles(("xyz", "type", "h"))
    off, nb = gpu.neighbors()
    tets, q = gpu.Reconstruct_tets()
    gpu.close()
    ot, oq = oracle.tetrahedralize(p["xyz"], p["type"], p["h"], off, nb, case.params["cutoff"],
                                   case.params["box_l"], case.params["box_r"])
    assert np.array_equal(tets, ot)
    for k in ("ntet", "nopen", "ndeleted", "ntie", "ntrunc"):
        assert q[k] == oq[k], k
    return len(ot)


@pytest.mark.parametrize("kind,side", [("jitter", 6), ("random", 6), ("lattice", 5), ("jitter", 8)])
@pytest.mark.parametrize("power", [-22, -25, -28, -32, -37])
def test_close_particles(kind, side, power):
    n = _check(_lattice(kind, 3, [1.0, 0.0, 0.0], 2.0 ** power, side))
    assert n > 0 or kind == "lattice"  # a lattice's spheres hold more than four points


@pytest.mark.parametrize("power", [-20, -30, -40])
def test_twins(power):
    x = _lattice("jitter", 3, [1.0, 0.0, 0.0], 1 / 32, 6)
    d = np.random.default_rng(5).normal(size=x.shape)
    assert _check(np.concatenate([x, x + 2.0 ** power * d])) > 0
