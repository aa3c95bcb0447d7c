"""Triangles of particles so close together, or of bodies so large, that FP32 cannot
hold the products of two of their lengths, against the oracle on the same
particles and rows.  (Beyond 2^68 the neighbour search's own FP32 squares
overflow.)"""
import pytest

from mrsph import SPHMeshGeneration, cases
from test_gpu_mesh_paths import _lattice
from test_gpu_tri import _compare

pytestmark = pytest.mark.gpu


def _mesh(case, xyz):
    gpu = SPHMeshGeneration(case, precision="fp64", neighbor_cap=1000)
    gpu.set_state({"xyz": xyz})
    gpu.run_phase(3)
    tris, q = _compare(gpu, case)
    gpu.close()
    assert len(tris) > 144


@pytest.mark.parametrize("kind", ["jitter", "random"])
@pytest.mark.parametrize("power", [-70, -66, -62, -58, -54, -44, -36])
def test_close_particles(kind, power):
    """Around the origin, where FP64 coordinates hold such spacings, inside the body."""
    case = cases.disc_hole_2d(spacing=0.02, grid=64)
    shift = [0.17, 0.21, 0.0]
    for k in ("box_l", "box_r"):
        case.params[k] = [v - t for v, t in zip(case.params[k], shift)]
    for lv in case.levels:
        lv.box_l = [v - t for v, t in zip(lv.box_l, shift)]
    _mesh(case, _lattice(kind, 2, [0.0, 0.0, 0.0], 2.0 ** power, 12))


@pytest.mark.parametrize("kind", ["jitter", "random"])
@pytest.mark.parametrize("power", [40, 58, 66, 68])
def test_large_bodies(kind, power):
    case = cases.disc_hole_2d(spacing=0.02, grid=64)
    s, p = 2.0 ** power, case.params
    for k in ("min_dl", "max_dl"):
        p[k] *= s
    for k in ("box_l", "box_r"):
        p[k] = [v * s for v in p[k]]
    for lv in case.levels:
        lv.phi = lv.phi * s
        lv.box_l, lv.dpkg = [v * s for v in lv.box_l], [v * s for v in lv.dpkg]
    _mesh(case, _lattice(kind, 2, [0.17, 0.21, 0.0], 0.0156, 12) * s)
