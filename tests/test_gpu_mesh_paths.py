"""The mesh passes where their FP32 decisions and tile sizes end: neighbour rows
shorter and longer than the rows kept in shared memory, lattices (every
predicate is zero somewhere: the exact signs decide), nearly flat point sets
and dense random ones, against the oracle on the same particles and rows."""
import numpy as np
import pytest

import oracle
from mrsph import SPHMeshGeneration, cases
from test_gpu_tri import _compare

pytestmark = pytest.mark.gpu


def _lattice(kind, dim, centre, spacing, side):
    g = (np.arange(side) - side / 2) * spacing
    x = np.stack([v.ravel() for v in np.meshgrid(*[g] * dim, indexing="ij")], 1)
    rng = np.random.default_rng(side)
    if kind == "jitter":
        x = x + rng.uniform(-0.3, 0.3, x.shape) * spacing
    elif kind == "thin":  # close to a lattice: side tests and spheres near their bounds
        x = x + rng.uniform(-1e-6, 1e-6, x.shape) * spacing
    elif kind == "random":
        x = rng.uniform(-0.5, 0.5, x.shape) * spacing * side
    out = np.zeros((len(x), 3))
    out[:, :dim] = x
    return out + centre


@pytest.mark.parametrize("kind", ["lattice", "thin", "jitter", "random"])
@pytest.mark.parametrize("cap", [64, 1000, 9000])
def test_tri_row_lengths(kind, cap):
    """9000 entries a row do not fit a warp's shared memory: every slot is then
    decided exactly."""
    case = cases.disc_hole_2d(spacing=0.02, grid=64)
    gpu = SPHMeshGeneration(case, precision="fp64", neighbor_cap=cap)
    gpu.set_state({"xyz": _lattice(kind, 2, [0.17, 0.21, 0.0], 0.0156 if cap > 64 else 0.02, 12)})
    gpu.run_phase(3)
    _compare(gpu, case)
    gpu.close()


@pytest.mark.parametrize("kind,spacing,side", [("lattice", 1 / 32, 6), ("thin", 1 / 32, 7), ("jitter", 1 / 32, 9),
                                               ("random", 1 / 40, 10), ("jitter", 1 / 64, 12)])
def test_tet_rows(kind, spacing, side):
    case = cases.torus_3d(dx_min=0.03, dx_max=0.09, fine_pkg=32, nlevels=2)
    gpu = SPHMeshGeneration(case, precision="fp64", neighbor_cap=2048)
    gpu.set_state({"xyz": _lattice(kind, 3, [1.0, 0.0, 0.0], spacing, side)})
    gpu.run_phase(3)
    p = gpu.particles(("xyz", "type", "h"))
    off, nb = gpu.neighbors()
    if spacing < 1 / 60:
        assert np.diff(off).max() > 256  # rows longer than the part kept in shared memory
    tets, q = gpu.Reconstruct_tets()
    gpu.close()
    ot, oq = oracle.tetrahedralize(p["xyz"], p["type"], p["h"], off, nb, case.params["cutoff"],
                                   case.params["box_l"], case.params["box_r"])
    assert np.array_equal(tets, ot)
    for k in ("ntet", "nopen", "ndeleted", "ntie", "ntrunc"):
        assert q[k] == oq[k], k
    for k in ("nsmall_dihedral", "aspect_hist", "radius_hist", "dihedral_hist"):
        assert list(q[k]) == list(oq[k]), k
