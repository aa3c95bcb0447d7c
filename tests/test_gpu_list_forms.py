"""The list and force forms (lanes and groups per particle, warp tiles, tiles in
brick order) on both sides of every dispatch line, alone and beside other
handles: a handle stepped alone, in the persistent batch kernel and on streams
has the same bits, and one step of a graded 3D body of each form matches the
oracle."""
import math

import numpy as np
import pytest

import oracle
from mrsph import BatchRelaxation, SPHMeshGeneration, cases
from paritylib import gpu_post_map_to_oracle, warm_oracle
from test_gpu_parity import _gpu_step_taps, check_fp32_single_step

pytestmark = pytest.mark.gpu

FIELDS = ("xyz", "type", "h", "sum")


def star(dim, n):
    case = cases.star_shape(dim, 5, n)
    case.n_particles = n
    return case


def graded2(n):
    dx = 0.001 * math.sqrt(77551.0 / n)
    case = cases.ellipses_2d(n_ellipses=8, dx_min=dx, dx_max=8 * dx, grid=128)
    case.n_particles = n
    return case


def graded3(n, target):
    """A torus whose spacing fits target particles, seeded with n: rows of about 280 n / target neighbours."""
    dx = 0.005 * (2410164.0 / target) ** (1 / 3.0)
    for _ in range(200):  # the spacing range has to give a consistent cell-list plan
        try:
            case = cases.torus_3d(dx_min=dx, dx_max=4 * dx, fine_pkg=32, nlevels=2)
            break
        except ValueError:
            dx *= 1.003
    case.n_particles = n
    return case


BODIES = {
    "2d_24576": lambda: star(2, 24576), "2d_24577": lambda: star(2, 24577),
    "graded2d_73728": lambda: graded2(73728), "graded2d_73729": lambda: graded2(73729),
    "3d_57344": lambda: star(3, 57344), "3d_57345": lambda: star(3, 57345),
    "graded3d_98304": lambda: graded3(98304, 400000), "graded3d_98305": lambda: graded3(98305, 400000),
    "graded3d_196608": lambda: graded3(196608, 800000), "graded3d_196609": lambda: graded3(196609, 800000),
    "dense3d_49152": lambda: graded3(49152, 49152), "dense3d_49153": lambda: graded3(49153, 49153),
}


def stepped(case, how, steps=4, beside=None):
    hs = [SPHMeshGeneration(c, precision="fp32") for c in [case] + ([beside] if beside else [])]
    for h in hs:
        h.Initialize_case()
    if how == "alone":
        for h in hs:
            h.SPH_run_mesh_generation(steps)
    else:
        b = BatchRelaxation(hs, mode=how)
        b.SPH_run_mesh_generation(steps)
        b.sync()
        b.close()
    out = hs[0].particles(FIELDS), hs[0].stats()["pairs"]
    for h in hs:
        h.close()
    return out


def same(a, b):
    assert a[1] == b[1]
    for k in FIELDS:
        assert np.array_equal(a[0][k], b[0][k]), k


@pytest.mark.parametrize("body", list(BODIES))
def test_alone_equals_batch(body):
    case = BODIES[body]()
    a = stepped(case, "alone")
    row = a[1] / case.n_particles
    assert (row > 160) == body.startswith("dense")
    same(a, stepped(case, "persistent"))


@pytest.mark.parametrize("small,big", [(star(2, 3000), star(2, 80000)), (star(3, 4000), star(3, 60000)),
                                       (graded3(6000, 12000), star(3, 100000))], ids=["2d", "3d", "graded3d"])
def test_beside_a_large_handle(small, big):
    """On streams a small handle takes the forms of the whole batch's size."""
    a = stepped(small, "alone")
    same(a, stepped(small, "streams", beside=big))
    same(a, stepped(small, "streams"))


@pytest.mark.parametrize("n,target", [(98305, 98305), (98305, 400000), (196609, 800000)],
                         ids=["dense tiles", "tiles", "bricks"])
def test_graded_step_matches_oracle(n, target):
    case = graded3(n, target)
    st = warm_oracle(case, max_steps=1, need_surface=False).get_state()
    assert len(st["x"]) == n
    check_fp32_single_step(case, st)


@pytest.mark.parametrize("dim,side,target", [(2, 160, 60000), (3, 40, 200000)])
def test_pairs_on_the_cut_off(dim, side, target):
    """A lane decides in FP32 and leaves a particle with a pair in the criterion's
    band to a group: a lattice whose spacing divides the cut-off radius, so that
    nearly every particle has such pairs."""
    case = star(dim, target)
    case.n_particles = n = side ** dim
    p = case.params
    st = warm_oracle(case, max_steps=1, need_surface=False).get_state()
    g = (np.arange(side) - side / 2) * (p["min_dl"] * p["cell_ratio"] / (3.0 if dim == 2 else 2.0))
    axes = [v.ravel() for v in np.meshgrid(*[g] * dim, indexing="ij")]
    for d, k in enumerate("xyz"):
        st[k] = axes[d] + 0.5 * (p["box_l"][d] + p["box_r"][d]) if d < dim else np.zeros(n)
        st["v" + k] = np.zeros(n)
    gp, lc, ids, off, nb, stats = _gpu_step_taps(case, "fp32", st)
    o2 = oracle.Oracle(case)
    gpu_post_map_to_oracle(o2, gp, st)
    ooff, onb = o2.neighbors()
    assert np.array_equal(off, ooff) and np.array_equal(nb, onb)
