"""Levels refined from their grandparent's state (grand.cuh) against the
oracle, bit for bit (0 ulp: same formulas, same order): closed inputs whose
grandparent mesh has faces of 3 to 8 corners (summed by the face's first
corner), 9 (k_g3, one thread), 17 and 64 (k_g3, a warp) and 65; as the last
level and as one that writes the next level's state; fewer corners than one
block and not a multiple of one.  With compensated sums, against the general
path."""
import numpy as np
import pytest

import oracle
from slak_b200 import _abi, api, meshgen
from slak_b200.mesh import LAK, SLAK, from_arrays

pytestmark = pytest.mark.gpu


def _prism(n):
    """n quads between two n-gons: a closed mesh of valence 3."""
    a = 2 * np.pi * np.arange(n) / n
    xyz = np.concatenate([np.stack([np.cos(a), np.sin(a), np.full(n, z) + 0.01 * np.cos(3 * a)], 1) for z in (0, 1)])
    k = np.arange(n)
    quads = np.stack([k, (k + 1) % n, n + (k + 1) % n, n + k], 1)
    ids = np.concatenate([quads.ravel(), k[::-1], n + k])
    ptr = np.concatenate([4 * np.arange(n + 1), [5 * n, 6 * n]])
    return from_arrays(ptr, ids, xyz)


def _tetra():
    xyz = np.array([[1, 1, 1], [-1, -1, 1], [-1, 1, -1], [1, -1, -1]], np.float32)
    return from_arrays(np.arange(0, 13, 3), np.array([0, 1, 2, 0, 3, 1, 0, 2, 3, 1, 3, 2]), xyz)


MESHES = {"tetra": _tetra, "prism3": lambda: _prism(3), "cube": lambda: _prism(4), "prism8": lambda: _prism(8),
          "prism9": lambda: _prism(9), "prism17": lambda: _prism(17), "prism64": lambda: _prism(64),
          "prism65": lambda: _prism(65), "torus": lambda: meshgen.torus(11, 7, seed=4),
          "mixed": lambda: meshgen.mixed_torus(23, 19, 0.1, 0.1, 0.005, seed=6)}


def _same(a, b):
    assert np.array_equal(a.ids, b.ids)
    assert np.array_equal(np.asarray(a.verts, np.float32).view(np.uint32), np.asarray(b.verts, np.float32).view(np.uint32))


@pytest.mark.parametrize("scheme", [SLAK, LAK])
@pytest.mark.parametrize("levels", [3, 4, 5])
@pytest.mark.parametrize("name", MESHES)
def test_grandparent_levels_equal_the_oracle(name, levels, scheme):
    m = MESHES[name]()
    got, ref = api.subdivide(m, levels, scheme), oracle.subdivide(m, levels, scheme)
    _same(got, ref)
    if scheme == LAK:
        assert np.array_equal(got.ptr, ref.ptr) and np.array_equal(got.vals, ref.vals)
    _same(api.subdivide(m, levels, scheme, _abi.PLAN_COMPENSATED),
          api.subdivide(m, levels, scheme, _abi.PLAN_COMPENSATED | _abi.PLAN_GENERAL))


@pytest.mark.parametrize("scheme", [SLAK, LAK])
def test_grandparent_levels_in_groups(scheme):
    """The same meshes in one batch: grouped launches of each kernel."""
    ms = [MESHES[k]() for k in MESHES]
    b = api.Batch([api.DeviceMesh.from_host(m) for m in ms], [3 + i % 2 for i in range(len(ms))], scheme)
    b.execute()
    b.check()
    for i, m in enumerate(ms):
        _same(b.output(i).to_host(), oracle.subdivide(m, 3 + i % 2, scheme))
    b.close()
