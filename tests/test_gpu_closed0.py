"""Level 0 of closed meshes (closed0.cuh) against the oracle, bit for bit (0
ulp: same formulas, same order): valences at the edges of its paths (4, 8: one
thread; 9: records bucketed, one thread's vertex point; 16, 17, 64: a warp's;
65), faces of 8 and 9 corners, vertex counts around the four scan tiles one
launch covers, alone and before a level that reads its state.  Compensated
sums, and creases on the slot-ordered columns, against the general path."""
import numpy as np
import pytest

import oracle
from slak_b200 import _abi, api, meshgen
from slak_b200.mesh import LAK, SLAK, from_arrays
from test_gpu_grand import _prism, _same

pytestmark = pytest.mark.gpu


def _bipyramid(n):
    """2n triangles: two apices of valence n, a ring of valence 4."""
    a = 2 * np.pi * np.arange(n) / n
    xyz = np.concatenate([np.stack([np.cos(a), np.sin(a), 0.02 * np.sin(5 * a)], 1), [[0, 0, 1.0], [0, 0, -1.0]]])
    k = np.arange(n)
    up = np.stack([k, (k + 1) % n, np.full(n, n)], 1)
    down = np.stack([(k + 1) % n, k, np.full(n, n + 1)], 1)
    return from_arrays(3 * np.arange(2 * n + 1), np.concatenate([up, down]).ravel(), xyz)


MESHES = {f"bipyramid{n}": (lambda n=n: _bipyramid(n)) for n in (3, 4, 5, 8, 9, 16, 17, 64, 65)}
MESHES.update({f"prism{n}": (lambda n=n: _prism(n)) for n in (3, 4, 8, 9)})
MESHES.update({f"torus{w}x{h}": (lambda w=w, h=h: meshgen.torus(w, h, seed=w)) for w, h in ((4, 3), (91, 90), (128, 64), (83, 99))})
MESHES["mixed"] = lambda: meshgen.mixed_torus(37, 31, 0.1, 0.1, 0.005, seed=6)


@pytest.mark.parametrize("scheme", [SLAK, LAK])
@pytest.mark.parametrize("levels", [1, 2])
@pytest.mark.parametrize("name", MESHES)
def test_closed_level0_equals_the_oracle(name, levels, scheme):
    m = MESHES[name]()
    got, ref = api.subdivide(m, levels, scheme), oracle.subdivide(m, levels, scheme)
    _same(got, ref)
    if scheme == LAK:
        assert np.array_equal(got.ptr, ref.ptr) and np.array_equal(got.vals, ref.vals)
    C = _abi.PLAN_COMPENSATED
    _same(api.subdivide(m, levels, scheme, C), api.subdivide(m, levels, scheme, C | _abi.PLAN_GENERAL))


@pytest.mark.parametrize("scheme", [SLAK, LAK])
@pytest.mark.parametrize("name", ["bipyramid8", "bipyramid17", "mixed"])
def test_creases_on_a_closed_level0(name, scheme):
    m = MESHES[name]()
    a, b = m.ids, m.ids[np.concatenate([np.r_[np.arange(s + 1, e), s] for s, e in zip(m.ptr[:-1], m.ptr[1:])])]
    some = np.flatnonzero(a < b)[::3]
    creases = (np.stack([a[some], b[some]], 1), np.linspace(0.5, 2.5, some.size).astype(np.float32))
    _same(api.subdivide(m, 3, scheme, creases=creases), api.subdivide(m, 3, scheme, _abi.PLAN_GENERAL, creases=creases))
