"""Face offsets that describe no mesh (overlapping many times over, out of range,
leaving corners out) are refused by every entry point with SLAK_ERR_BAD_MESH; the
level-0 topology pass that finds them keeps to its arrays, and a sound mesh is
refined as before afterwards."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from slak_b200 import _abi, api, meshgen
from slak_b200.mesh import LAK, SLAK
from test_gpu_grand import _same

pytestmark = pytest.mark.gpu

BAD = 4                                             # SLAK_ERR_BAD_MESH


def _offsets(kind, ptr):
    p, n = ptr.astype(np.int64).copy(), int(ptr[-1])
    if kind == "overlapping":                       # every other face is the whole mesh
        p[:] = np.where(np.arange(p.size) % 2, n, 0)
    elif kind == "beyond":
        p[5:-1:3] += 1 << 30
    elif kind == "negative":
        p[5:-1:3] = -7
    elif kind == "first":
        p[0] = 1 << 30
    elif kind == "tail":                            # the last faces' corners in no face
        p[-6:] = p[-7]
    return p.astype(np.int32)


KINDS = ["overlapping", "beyond", "negative", "first", "tail"]


@pytest.mark.parametrize("scheme", [SLAK, LAK])
@pytest.mark.parametrize("kind", KINDS)
def test_bad_offsets_are_refused(kind, scheme):
    lib = _abi.lib()
    good = meshgen.mixed_torus(24, 20, 0.1, 0.06, 0.005, seed=5)
    bad = good.copy()
    bad.ptr = _offsets(kind, np.asarray(good.ptr))
    dm = api.DeviceMesh.from_host(bad)
    c, out = dm.as_c(), _abi.SlakMesh()
    for flags in (0, _abi.PLAN_GENERAL):
        with pytest.raises(_abi.SlakError) as e:
            api.Plan(dm, 2, scheme, flags)
        assert e.value.code == BAD
    assert lib.slak_subdivide(ctypes.byref(c), ctypes.byref(out), 2, scheme, None) == BAD
    with pytest.raises(_abi.SlakError) as e:
        api.Batch([api.DeviceMesh.from_host(good), dm], [1, 2], scheme)
    assert e.value.code == BAD
    ids = torch.empty(16 * bad.nnz, dtype=torch.int32, device="cuda")
    verts = torch.empty(4 * (bad.nverts + bad.nfaces + bad.nnz), dtype=torch.float32, device="cuda")
    r = _abi.SlakMesh()
    r.nverts = verts.numel() // 4
    r.ids, r.verts = ids.data_ptr(), verts.data_ptr()
    r.ptr, r.vals = ids.data_ptr(), ids.data_ptr()  # (never written: the call is refused)
    assert lib.slak_subdivide_level_noalloc(ctypes.byref(c), ctypes.byref(r), scheme, None) == BAD
    torch.cuda.synchronize()
    _same(api.subdivide(good, 2, scheme), oracle.subdivide(good, 2, scheme))
