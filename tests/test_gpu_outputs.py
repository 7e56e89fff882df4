"""Output arrays kept between one-shot calls: a result that is still held is
never handed out again, a released one may be, results stay those of the
oracle, slak_workspace_release gives the memory back, and arrays the caller
freed with cudaFree are simply gone."""
import ctypes
import glob
import os

import numpy as np
import pytest
import torch

import oracle
from slak_b200 import _abi, api, meshgen
from slak_b200.mesh import LAK, SLAK

pytestmark = pytest.mark.gpu

CALL = {SLAK: api.CatmullClark, LAK: api.LAKCatmullClark}


def _refine(dm, scheme, levels):
    out = api.DeviceMesh()
    CALL[scheme].subdivideIteratively(dm, out, levels)
    return out


def _check(out, ref):
    assert np.array_equal(out.ids.cpu().numpy(), ref.ids)
    assert np.array_equal(out.verts.cpu().numpy().view(np.uint32), ref.verts.reshape(-1).view(np.uint32))


@pytest.mark.parametrize("scheme", [SLAK, LAK])
def test_released_outputs_are_reused_and_held_ones_are_not(scheme):
    assert _abi.lib().slak_workspace_release() == _abi.SLAK_OK
    m, small = meshgen.torus(40, 30, seed=2), meshgen.torus(11, 9, seed=3)
    ref, ref_small = oracle.subdivide(m, 2, scheme), oracle.subdivide(small, 2, scheme)
    dm, ds = api.DeviceMesh.from_host(m), api.DeviceMesh.from_host(small)
    a, b = _refine(dm, scheme, 2), _refine(dm, scheme, 2)
    pointers = lambda r: {t.data_ptr() for t in (r.ids, r.verts, r.ptr, r.vals) if t is not None}
    held, released = pointers(a), pointers(b)
    assert held.isdisjoint(released)
    del b
    c = _refine(dm, scheme, 2)
    assert pointers(c) == released
    s = _refine(ds, scheme, 2)
    for out, r in ((a, ref), (c, ref), (s, ref_small)):
        _check(out, r)
    del a, c, s
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    assert _abi.lib().slak_workspace_release() == _abi.SLAK_OK
    assert torch.cuda.mem_get_info()[0] >= before
    _check(_refine(dm, scheme, 2), ref)


def test_arrays_freed_with_cudafree():
    import nvidia.cuda_runtime
    so = glob.glob(os.path.join(list(nvidia.cuda_runtime.__path__)[0], "lib", "libcudart.so*"))[0]
    cudart = ctypes.CDLL(so)
    dm = api.DeviceMesh.from_host(meshgen.torus(16, 12, seed=5))
    ref = oracle.subdivide(meshgen.torus(16, 12, seed=5), 2, SLAK)
    for _ in range(3):
        cin, c = dm.as_c(), _abi.SlakMesh()
        assert _abi.lib().slak_subdivide(ctypes.byref(cin), ctypes.byref(c), 2, SLAK, None) == _abi.SLAK_OK
        assert cudart.cudaFree(ctypes.c_void_p(c.verts)) == 0
        c.verts = None
        assert _abi.lib().slak_mesh_free(ctypes.byref(c)) == _abi.SLAK_OK
        _check(_refine(dm, SLAK, 2), ref)


def test_no_cache_in_the_environment(monkeypatch):
    monkeypatch.setenv("SLAK_WORKSPACE_CACHE", "0")
    m = meshgen.torus(16, 12, seed=6)
    _check(_refine(api.DeviceMesh.from_host(m), SLAK, 2), oracle.subdivide(m, 2, SLAK))
