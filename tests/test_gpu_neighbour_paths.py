"""The neighbour passes on both sides of their dispatch lines (particles per
handle up to which a group of lanes takes one particle: 40,960 in the force
passes, 98,304 in 2D and 114,688 in 3D in the list builder) and the cell scan with more than 2048
blocks: one step against the oracle, and a handle alone against the persistent
batch kernel, which has one form for every size."""
import numpy as np
import pytest

import oracle
from mrsph import BatchRelaxation, SPHMeshGeneration, cases
from paritylib import gpu_post_map_to_oracle, rel_err, warm_oracle
from test_gpu_parity import _gpu_step_taps, check_fp32_single_step

pytestmark = pytest.mark.gpu

EDGES = [40960, 40961, 98304, 98305, 114688, 114689]


def sized_star(dim, n, n_target=None):
    case = cases.star_shape(dim, 5, n_target or n)
    case.n_particles = n
    return case


@pytest.mark.parametrize("n", EDGES)
@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_single_step(n, prec):
    case = sized_star(2, n)
    st = warm_oracle(case, max_steps=1, need_surface=False).get_state()
    assert len(st["x"]) == n
    if prec == "fp32":
        check_fp32_single_step(case, st)
        return
    gp, lc, ids, off, nb, stats = _gpu_step_taps(case, prec, st)
    o2 = oracle.Oracle(case)
    gpu_post_map_to_oracle(o2, gp, st)
    ooff, onb = o2.neighbors()
    assert np.array_equal(off, ooff) and np.array_equal(nb, onb)
    o2.density(ooff, onb)
    assert rel_err(gp["sum"], o2.get_state()["sum"]) < 1e-12
    o2.force(ooff, onb, 1)
    s1 = o2.get_state()
    assert rel_err(gp["a1"], np.stack([s1["ax"], s1["ay"], s1["az"]], 1)) < 1e-12
    o2.force(ooff, onb, 2)
    s2 = o2.get_state()
    assert rel_err(gp["a2"], np.stack([s2["ax"], s2["ay"], s2["az"]], 1), floor=1e-300) < 1e-12


@pytest.mark.parametrize("n", EDGES)
@pytest.mark.parametrize("dim", [2, 3])
def test_solo_equals_batch(n, dim):
    case = sized_star(dim, n)
    out = []
    for batched in (False, True):
        g = SPHMeshGeneration(case, precision="fp32")
        g.Initialize_case()
        if batched:
            b = BatchRelaxation([g])
            b.set_mode("persistent")
            b.SPH_run_mesh_generation(3)
            b.close()
        else:
            g.SPH_run_mesh_generation(3)
        out.append(g.particles(("xyz", "type", "h", "sum")))
        g.close()
    for k in ("xyz", "type", "h", "sum"):
        assert len(out[0][k]) == n
        assert np.array_equal(out[0][k], out[1][k]), k


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_scan_of_many_cells(prec):
    case = sized_star(2, 3000, n_target=16_000_000)  # some 26 million half cells
    st = warm_oracle(case, max_steps=1, need_surface=False).get_state()
    gp, lc, ids, off, nb, stats = _gpu_step_taps(case, prec, st)
    o2 = oracle.Oracle(case)
    gpu_post_map_to_oracle(o2, gp, st)
    assert np.array_equal(lc, o2.cells())
    ooff, onb = o2.neighbors()
    assert np.array_equal(off, ooff) and np.array_equal(nb, onb)
    assert np.array_equal(np.sort(ids), np.arange(3000))
