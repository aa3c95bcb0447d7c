"""A list capacity that grows after a step keeps that step's neighbour lists: the
lists read afterwards, and a mesh built from them, equal those of a handle
whose capacity was large from the start, alone and in a batch."""
import numpy as np
import pytest

from mrsph import BatchRelaxation, SPHMeshGeneration, cases

pytestmark = pytest.mark.gpu


def crowded(dim, n):
    """n particles, uniformly random: rows several times longer than relaxed ones."""
    case = cases.star_shape(dim, 6, n // 4)
    case.n_particles = n
    return case


def relaxed(case, how, steps, **kw):
    g = SPHMeshGeneration(case, precision="fp32", **kw)
    g.Initialize_case()
    if how == "solo":
        g.SPH_run_mesh_generation(steps)
    else:
        b = BatchRelaxation([g])
        b.set_mode(how)
        b.SPH_run_mesh_generation(steps)
        b.close()
    return g


@pytest.mark.parametrize("dim,n", [(2, 4000), (3, 6000)])
@pytest.mark.parametrize("how", ["solo", "persistent", "streams"])
def test_lists_survive_growth(dim, n, how):
    case = crowded(dim, n)
    steps = 1 if how == "solo" else 32  # the steps after which the capacity is checked
    ref = relaxed(case, "solo", steps, neighbor_cap=2048)
    got = relaxed(case, how, steps)
    try:
        r, q = ref.neighbors(), got.neighbors()
        assert np.array_equal(r[0], q[0]) and np.array_equal(r[1], q[1])
        assert ref.stats()["pairs"] == got.stats()["pairs"]
        mesh = (lambda s: s.Reconstruct_tris()) if dim == 2 else (lambda s: s.Reconstruct_tets())
        a, b = mesh(ref), mesh(got)
        assert len(a[0]) > 0 and np.array_equal(a[0], b[0])
    finally:
        ref.close()
        got.close()
