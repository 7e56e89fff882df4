"""Every launch shape the autotuner may pick for the levels of closed meshes gives
the oracle's bits: the nine pairs of k_p1's block size and register cap, as the
last level and as one that writes its state, k_pp from a polygon and a quad
grandparent, likewise, and k_g1 of a closed quad mesh, also where the next level
makes its quads unnecessary.  Each shape is forced through a SLAK_TUNE_FILE (read
once per process: one child process a shape)."""
import json
import os
import subprocess
import sys

import pytest

from slak_b200 import api, meshgen
from slak_b200.mesh import LAK, SLAK

pytestmark = pytest.mark.gpu

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CASES = [("mixed", 2), ("mixed", 3), ("mixed", 5), ("torus", 2), ("torus", 3), ("torus", 5)]


def mesh(name, scheme):
    m = meshgen.mixed_torus(13, 11, 0.1, 0.1, 0.005, seed=31) if name == "mixed" else meshgen.torus(13, 11, seed=32)
    return m.with_quad_ptr() if scheme == LAK and m.ptr is None else m


CHILD = r"""
import json, sys
sys.path[:0] = [sys.argv[1], sys.argv[1] + "/tests"]
import numpy as np
import oracle
from slak_b200 import api
from slak_b200.mesh import LAK, SLAK
from test_gpu_launch_shapes import CASES, mesh
rows = []
for name, levels in CASES:
    for scheme in (SLAK, LAK):
        m = mesh(name, scheme)
        plan = api.Plan(api.DeviceMesh.from_host(m), levels, scheme, 0)
        plan.execute()
        plan.check()
        out, ref = plan.output().to_host(), oracle.subdivide(m, levels, scheme)
        blocks = [t["block"] for t in plan.tuning() if t["state"] >= 0]
        plan.close()
        same = (np.array_equal(out.ids, ref.ids)
                and np.array_equal(np.asarray(out.verts, np.float32).view(np.uint32), ref.verts.view(np.uint32)))
        if scheme == LAK:
            same = same and np.array_equal(out.ptr, ref.ptr) and np.array_equal(out.vals, ref.vals)
        rows.append({"case": [name, levels, scheme], "same": bool(same), "blocks": blocks})
print(json.dumps(rows))
"""


@pytest.mark.parametrize("b1", [128, 256, 512])
@pytest.mark.parametrize("b0", [128, 256, 512])
def test_every_launch_shape_of_closed_levels(b0, b1, tmp_path):
    keys = set()
    for name, levels in CASES:
        for scheme in (SLAK, LAK):
            plan = api.Plan(api.DeviceMesh.from_host(mesh(name, scheme)), levels, scheme, 0)
            keys |= {t["key"] for t in plan.tuning() if t["state"] >= 0}
            plan.close()
    assert {k.split("/")[1] for k in keys} == {"poly1", "pppoly", "ppquad", "quad"}
    b2 = {128: 512, 256: 128, 512: 256}[b0]
    path = tmp_path / "tune.txt"
    path.write_text("".join(f"{k} {b0} {b1} {b2}\n" for k in sorted(keys)))
    r = subprocess.run([sys.executable, "-c", CHILD, REPO], env=dict(os.environ, SLAK_TUNE_FILE=str(path)),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
    rows = json.loads(r.stdout.strip().splitlines()[-1])
    assert len(rows) == 2 * len(CASES)
    for row in rows:
        assert row["same"], row
        assert row["blocks"] and all(b == [b0, b1, b2] for b in row["blocks"]), row
