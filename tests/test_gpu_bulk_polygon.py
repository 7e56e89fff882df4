"""SLAK_PLAN_BULK_RECORDS holds for every closed level, the first one after a
closed polygon input too: its k_g3 stages its records by bulk copy (a spent poll
budget is reported), and gives the default path's and the oracle's bits."""
import numpy as np
import pytest

import oracle
from slak_b200 import _abi, api, meshgen
from slak_b200.mesh import LAK, SLAK
from test_gpu_grand import _prism, _same

pytestmark = pytest.mark.gpu

MESHES = {"mixed": lambda: meshgen.mixed_torus(64, 48, 0.05, 0.03, 0.005, seed=8), "prism17": lambda: _prism(17)}


@pytest.mark.parametrize("scheme", [SLAK, LAK])
@pytest.mark.parametrize("levels", [2, 3])
@pytest.mark.parametrize("name", MESHES)
def test_bulk_records_after_a_polygon_input(name, levels, scheme):
    m = MESHES[name]()
    got, ref = api.subdivide(m, levels, scheme, _abi.PLAN_BULK_RECORDS), oracle.subdivide(m, levels, scheme)
    _same(got, ref)
    if scheme == LAK:
        assert np.array_equal(got.ptr, ref.ptr) and np.array_equal(got.vals, ref.vals)


@pytest.mark.parametrize("scheme", [SLAK, LAK])
def test_a_spent_budget_is_reported_at_the_first_level(scheme, monkeypatch):
    dm = api.DeviceMesh.from_host(MESHES["mixed"]())
    monkeypatch.setenv("SLAK_BULK_WAIT_POLLS", "0")         # the first poll is never made
    p = api.Plan(dm, 2, scheme, _abi.PLAN_BULK_RECORDS)
    p.execute()
    assert p.status() == 5                                  # SLAK_ERR_TIMEOUT
    p.close()
