"""slak_mesh_free of a one-shot call's result: it waits for whatever still uses
the arrays, on any stream, as cudaFree does; and it may be called while another
thread captures a graph in thread-local mode, as cudaFree may, without failing
and without invalidating that capture."""
import ctypes
import threading

import numpy as np
import pytest
import torch

import oracle
from slak_b200 import _abi, api, meshgen
from slak_b200.mesh import SLAK

pytestmark = pytest.mark.gpu


def _call(dm, levels=2):
    cin, c = dm.as_c(), _abi.SlakMesh()
    _abi.check(_abi.lib().slak_subdivide(ctypes.byref(cin), ctypes.byref(c), levels, SLAK, None), "slak_subdivide")
    return c


def _free(c):
    return _abi.lib().slak_mesh_free(ctypes.byref(c))


def test_free_waits_for_work_on_other_streams():
    dm = api.DeviceMesh.from_host(meshgen.torus(16, 12, seed=1))
    s = torch.cuda.Stream()
    for _ in range(3):                              # the first wait and later ones
        c = _call(dm)
        torch.cuda.synchronize()
        with torch.cuda.stream(s):
            torch.cuda._sleep(10_000_000)           # about 5 ms
        assert not s.query()
        assert _free(c) == _abi.SLAK_OK
        assert s.query()


def test_free_beside_another_threads_capture():
    m = meshgen.torus(16, 12, seed=1)
    dm = api.DeviceMesh.from_host(m)
    results = [_call(dm) for _ in range(2)]
    torch.cuda.synchronize()
    x, rc = torch.zeros(16, device="cuda"), []
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode="thread_local"):
        x += 1
        t = threading.Thread(target=lambda: rc.extend(_free(c) for c in results))
        t.start()
        t.join()
        x += 1
    g.replay()
    torch.cuda.synchronize()
    assert rc == [_abi.SLAK_OK] * 2
    assert x.tolist() == [2.0] * 16
    # the freed arrays serve the next call
    out = api.DeviceMesh()
    api.CatmullClark.subdivideIteratively(dm, out, 2)
    ref = oracle.subdivide(m, 2, SLAK)
    assert np.array_equal(out.ids.cpu().numpy(), ref.ids)
    assert np.array_equal(out.verts.cpu().numpy().view(np.uint32), ref.verts.reshape(-1).view(np.uint32))


def _cudart():
    import glob
    import os
    import nvidia.cuda_runtime
    return ctypes.CDLL(glob.glob(os.path.join(list(nvidia.cuda_runtime.__path__)[0], "lib", "libcudart.so*"))[0])


def _allocation_size(p):
    base, size = ctypes.c_uint64(), ctypes.c_size_t()
    assert ctypes.CDLL("libcuda.so.1").cuMemGetAddressRange_v2(ctypes.byref(base), ctypes.byref(size),
                                                               ctypes.c_uint64(p)) == 0
    assert base.value == p
    return size.value


def test_an_address_that_was_freed_and_allocated_larger():
    """A result freed with cudaFree whose address comes back as another, larger
    array: slak_mesh_free of that one must not keep it under the old size."""
    lib, cudart = _abi.lib(), _cudart()
    dm = api.DeviceMesh.from_host(meshgen.torus(16, 12, seed=1))
    assert lib.slak_workspace_release() == _abi.SLAK_OK
    c = _call(dm)
    size, want = 4 * c.nnz, 4 * c.nnz + 32768       # (ids and verts are 48 KiB each, one behind the other)
    old = c.ids
    for p in (c.ids, c.verts):
        assert cudart.cudaFree(ctypes.c_void_p(p)) == 0
    again = []
    for _ in range(16):                             # the driver's first fit: usually the first
        p = ctypes.c_void_p()
        assert cudart.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(want)) == 0
        again.append(p.value)
        if p.value == old:
            break
    for p in again:
        m = _abi.SlakMesh()
        m.ids = p
        assert _free(m) == _abi.SLAK_OK
    n = _call(dm)
    assert _allocation_size(n.ids) == size and _allocation_size(n.verts) == 16 * n.nverts
    assert _free(n) == _abi.SLAK_OK


def test_a_second_free_is_an_error_and_harms_no_later_result():
    """A copied descriptor freed twice: the second free is refused (as cudaFree
    would), and the arrays kept by the first stay good for later calls."""
    m = meshgen.torus(16, 12, seed=1)
    dm, ref = api.DeviceMesh.from_host(m), oracle.subdivide(m, 2, SLAK)
    c = _call(dm)
    copy = _abi.SlakMesh.from_buffer_copy(c)
    assert _free(c) == _abi.SLAK_OK
    assert _free(copy) == 2                         # SLAK_ERR_CUDA
    outs = []
    for _ in range(2):
        out = api.DeviceMesh()
        api.CatmullClark.subdivideIteratively(dm, out, 2)
        outs.append(out)
    assert outs[0].ids.data_ptr() != outs[1].ids.data_ptr()
    for out in outs:
        assert np.array_equal(out.ids.cpu().numpy(), ref.ids)
        assert np.array_equal(out.verts.cpu().numpy().view(np.uint32), ref.verts.reshape(-1).view(np.uint32))
