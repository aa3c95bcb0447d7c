"""Results copied into the caller's arrays: level-set fields and samples written
at odd offsets of larger arrays leave what surrounds them alone, samples on
both sides of the size up to which they go through a host buffer agree, and the
points' own array may take the normals."""
import ctypes as C

import numpy as np
import pytest

from mrsph import SPHMeshGeneration, cases

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    g = SPHMeshGeneration(cases.torus_3d(dx_min=0.03, dx_max=0.09, fine_pkg=32, nlevels=2), precision="fp64")
    yield g
    g.close()


def at(a, k):
    return C.c_void_p(a.ctypes.data + k * a.itemsize)


def test_fields_at_odd_offsets(gpu):
    want = gpu.levelset_fields(1)
    n, odd, pad = gpu.case.levels[1].phi.size, 8191, 12345
    big = [np.full(n + pad, -7.25) for _ in range(4)]
    tag = np.full(n + pad, 201, np.uint8)
    rc = gpu.lib.mrsph_get_levelset(gpu.h, 1, *[at(a, odd) for a in big], at(tag, odd), None)
    assert rc == 0
    got = {"nx": big[0], "ny": big[1], "nz": big[2], "curv": big[3], "tag": tag}
    for k, a in got.items():
        assert np.array_equal(a[odd: odd + n], want[k].ravel()), k
        edge = 201 if k == "tag" else -7.25
        assert (a[:odd] == edge).all() and (a[odd + n:] == edge).all(), k


@pytest.mark.parametrize("n", [1, 5957, 5958, 70000])
def test_samples(gpu, n):
    rng = np.random.default_rng(n)
    lo, hi = np.array(gpu.case.params["box_l"]), np.array(gpu.case.params["box_r"])
    xyz = lo + rng.random((n, 3)) * (hi - lo)
    phi, nrm, curv, tag = gpu.sample_levelset(xyz)
    for k in range(0, n, 997):  # short calls
        p, m, c, t = gpu.sample_levelset(xyz[k: k + 997])
        assert np.array_equal(p, phi[k: k + 997]) and np.array_equal(m, nrm[k: k + 997])
        assert np.array_equal(c, curv[k: k + 997]) and np.array_equal(t, tag[k: k + 997])
    own, some = xyz.copy(), np.full(n + 3, 9, np.int32)
    rc = gpu.lib.mrsph_sample_levelset(gpu.h, n, at(own, 0), None, at(own, 0), None, at(some, 1))
    assert rc == 0
    assert np.array_equal(own, nrm) and np.array_equal(some[1: n + 1], tag)
    assert some[0] == 9 and (some[n + 1:] == 9).all()
