"""What an execution zeroes: the status word, level 0's counts and, for polygon
faces, its corner -> face map, whatever other levels run (read off the memset
nodes of a captured execution)."""
import ctypes

import pytest
import torch

from slak_b200 import _abi, api, meshgen
from slak_b200.mesh import LAK, SLAK

pytestmark = pytest.mark.gpu


class _Memset(ctypes.Structure):
    _fields_ = [("dst", ctypes.c_uint64), ("pitch", ctypes.c_size_t), ("value", ctypes.c_uint),
                ("element", ctypes.c_uint), ("width", ctypes.c_size_t), ("height", ctypes.c_size_t)]


def _memset_bytes(plan):
    cu = ctypes.CDLL("libcuda.so.1")
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        plan.execute()
    graph, n = ctypes.c_void_p(int(g.raw_cuda_graph())), ctypes.c_size_t()
    assert cu.cuGraphGetNodes(graph, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(graph, nodes, ctypes.byref(n)) == 0
    out = []
    for node in nodes:
        t, m = ctypes.c_int(), _Memset()
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(t)) == 0
        if t.value == 2:                            # CU_GRAPH_NODE_TYPE_MEMSET
            assert cu.cuGraphMemsetNodeGetParams(ctypes.c_void_p(node), ctypes.byref(m)) == 0
            out.append(m.element * m.width * m.height)
    return out


@pytest.mark.parametrize("scheme", [SLAK, LAK])
@pytest.mark.parametrize("levels", [1, 3])
@pytest.mark.parametrize("flags", [0, _abi.PLAN_GENERAL])
def test_an_execution_zeroes_no_more_than_it_needs(flags, levels, scheme):
    m = meshgen.mixed_torus(24, 20, 0.1, 0.1, 0.005, seed=6)
    plan = api.Plan(api.DeviceMesh.from_host(m), levels, scheme, flags)
    plan.execute()
    plan.check()
    sizes, stats = _memset_bytes(plan), plan.level_stats()
    plan.close()
    # closed: one 8-byte count per vertex; general: 4 bytes per vertex of each
    # general level and 4 per corner of the polygon level; 4 KiB for the status
    # word and the arrays' alignment
    need = 8 * m.nverts if flags == 0 else 4 * (m.nnz + sum(s["nverts"] for s in stats))
    assert 0 < sum(sizes) <= need + 4096, sizes
