"""The output arrays kept between one-shot calls do not count as used memory:
slak_workspace_release returns them to the device, and so do, of their own
accord, a plan and a batch that would not fit beside them."""
import ctypes

import numpy as np
import pytest
import torch

import oracle
from slak_b200 import _abi, api, meshgen
from slak_b200.mesh import SLAK

pytestmark = pytest.mark.gpu

MIB = 1 << 20


def _free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _idle(n):
    """One result of an n x n torus, dropped: its two arrays stay allocated, idle."""
    dm = api.DeviceMesh.from_host(meshgen.torus(n, n, seed=1))
    out = api.DeviceMesh()
    api.CatmullClark.subdivideIteratively(dm, out, 1)
    size = 4 * (out.ids.numel() + out.verts.numel())
    del out, dm
    return size


def test_release_returns_the_idle_arrays():
    lib = _abi.lib()
    assert lib.slak_workspace_release() == _abi.SLAK_OK
    small = api.DeviceMesh.from_host(meshgen.torus(16, 12, seed=1))
    kept = _idle(700)                               # 2 arrays of 31 MB
    torch.cuda.empty_cache()
    before = _free_bytes()
    out = api.DeviceMesh()
    api.CatmullClark.subdivideIteratively(small, out, 1)
    del out
    assert _free_bytes() >= before - 4 * MIB        # the small call took none of them, and freed none
    assert lib.slak_workspace_release() == _abi.SLAK_OK
    assert _free_bytes() >= before + kept


@pytest.fixture
def almost_full():
    """About 540 MB of idle arrays on a device with no more than `left` free."""
    hold = []
    lib = _abi.lib()

    def fill(left):
        assert lib.slak_workspace_release() == _abi.SLAK_OK
        kept = _idle(2048)
        torch.cuda.empty_cache()
        rest = _free_bytes() - left
        assert rest > 0
        hold.append(torch.empty(rest, dtype=torch.uint8, device="cuda"))
        assert _free_bytes() <= left + 4 * MIB
        return kept

    yield fill
    hold.clear()
    torch.cuda.empty_cache()
    lib.slak_workspace_release()


def _bits(a):
    return np.asarray(a, np.float32).reshape(-1).view(np.uint32)


def test_a_plan_that_fits_without_the_idle_arrays(almost_full):
    m = meshgen.torus(600, 500, seed=2)
    ref = oracle.subdivide(m, 1, SLAK)
    dm = api.DeviceMesh.from_host(m)
    for warm in range(2):                           # (modules and streams are loaded before memory is short)
        if warm:
            almost_full(24 * MIB)                   # less than the probe and the outputs take
        plan = api.Plan(dm, 1, SLAK)
        plan.execute()
        plan.check()
        got = plan.output()
        ids, verts = got.ids.cpu().numpy(), got.verts.cpu().numpy()
        plan.close()
    assert np.array_equal(ids, ref.ids) and np.array_equal(_bits(verts), _bits(ref.verts))


def test_a_batch_that_fits_without_the_idle_arrays(almost_full):
    ms = [meshgen.torus(600, 500, seed=2), meshgen.mixed_torus(300, 200, 0.05, 0.03, 0.005, seed=3)]
    refs = [oracle.subdivide(m, 1, SLAK) for m in ms]
    dms = [api.DeviceMesh.from_host(m) for m in ms]
    for warm in range(2):
        if warm:
            almost_full(2048 * MIB + 16 * MIB)      # 2 GiB stay free by the batch's rule; its outputs take 48 MB
        b = api.Batch(dms, [1, 1], SLAK)
        b.execute()
        b.check()
        got = [(b.output(i).ids.cpu().numpy(), b.output(i).verts.cpu().numpy()) for i in range(2)]
        b.close()
    for (ids, verts), ref in zip(got, refs):
        assert np.array_equal(ids, ref.ids) and np.array_equal(_bits(verts), _bits(ref.verts))
