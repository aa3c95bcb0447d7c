"""MRSPH_FLAG_NEIGHBOR_SPILL stands for particles that a force stage re-scanned:
not for lists that a state's first step takes again in a larger capacity, but
for those of a capacity that the caller fixed."""
import numpy as np
import pytest

from mrsph import SPHMeshGeneration, cases

pytestmark = pytest.mark.gpu
SPILL = 8


def crowded(dim, n):
    case = cases.star_shape(dim, 6, n // 4)
    case.n_particles = n
    return case


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("dim,n,cap", [(2, 4000, 64), (3, 6000, 192)])
def test_spill_flag(dim, n, cap, prec):
    for fixed, first in ((0, 0), (cap, SPILL)):
        g = SPHMeshGeneration(crowded(dim, n), precision=prec, neighbor_cap=fixed)
        g.Initialize_case()
        g.SPH_run_mesh_generation(1)
        assert g.stats()["flags"] & SPILL == first
        if not fixed:
            assert np.diff(g.neighbors()[0]).max() > cap  # of the capacity that a handle starts with
        g.SPH_run_mesh_generation(1)
        assert g.stats()["flags"] & SPILL == first
        g.close()
