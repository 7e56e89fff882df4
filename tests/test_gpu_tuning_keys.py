"""A tuning key names the kernels it was measured on: the one-launch level 1 of a
closed polygon mesh is not the level 1 of other meshes (whose entries, in files of
earlier builds, meant other kernels), and a level refined from a polygon
grandparent is not one refined from a quad grandparent of the same size."""
import pytest

from slak_b200 import _abi, api, meshgen
from slak_b200.mesh import LAK, POLY, SLAK

pytestmark = pytest.mark.gpu


def _keys(m, levels, scheme):
    plan = api.Plan(api.DeviceMesh.from_host(m), levels, scheme, 0)
    keys = [t["key"] for t in plan.tuning()]
    plan.close()
    return keys


@pytest.mark.parametrize("scheme", [SLAK, LAK])
def test_keys_name_the_kernels(scheme):
    quad = meshgen.torus(32, 32, seed=1)
    # the same corner counts and valences, as polygon faces
    poly = meshgen.torus(32, 32, seed=1).with_quad_ptr()
    poly.type = POLY
    if scheme == LAK:
        quad = quad.with_quad_ptr()
    kq, kp = _keys(quad, 4, scheme), _keys(poly, 4, scheme)
    assert kq[0] == kp[0] == ""
    assert kq[3] == kp[3]                           # level 3: both grandparents are quads
    assert kq[1] != kp[1] and kq[2] != kp[2]
    assert len(set(kq[1:] + kp[1:])) == 5
    old = "lak" if scheme == LAK else "slak"
    assert not any(k.startswith(f"{old}/poly/") or "/pp-" in k for k in kq + kp)
