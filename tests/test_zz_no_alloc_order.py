"""Order of the kernels of bt_round_noalloc, read from a captured round.

The phase kernels read the halo tables in their prologues, before they wait for
the kernel ahead of them, so the one launch that follows the table kernel must
depend on it fully (not programmatically); those after it may overlap.
"""
import ctypes

import numpy as np
import pytest
import torch

from licom4py_gpu_b200 import _native as N
from licom4py_gpu_b200.duogrid import make_consts
from licom4py_gpu_b200.fields import harmonic_state
from licom4py_gpu_b200.plan import BtPlan, CONST_NAMES

pytestmark = pytest.mark.gpu

FULL, PROGRAMMATIC = 0, 1  # cudaGraphDependencyType
RELAXED = 2                # cudaStreamCaptureModeRelaxed


class EdgeData(ctypes.Structure):  # cudaGraphEdgeData
    _fields_ = [("from_port", ctypes.c_ubyte), ("to_port", ctypes.c_ubyte), ("type", ctypes.c_ubyte),
                ("reserved", ctypes.c_ubyte * 5)]


def _captured_edges(stream, call):
    """(from, to, type) of every edge of the graph that ``call`` makes on ``stream``; nothing runs."""
    rt = ctypes.CDLL("libcudart.so.12")
    s, graph, count = ctypes.c_void_p(stream.cuda_stream), ctypes.c_void_p(), ctypes.c_size_t()
    assert rt.cudaStreamBeginCapture(s, RELAXED) == 0
    try:
        call()
    finally:
        end = rt.cudaStreamEndCapture(s, ctypes.byref(graph))
    assert end == 0
    assert rt.cudaGraphGetEdges_v2(graph, None, None, None, ctypes.byref(count)) == 0
    src, dst, data = (ctypes.c_void_p * count.value)(), (ctypes.c_void_p * count.value)(), (EdgeData * count.value)()
    assert rt.cudaGraphGetEdges_v2(graph, src, dst, data, ctypes.byref(count)) == 0
    assert rt.cudaGraphDestroy(graph) == 0
    return [(a, b, d.type) for a, b, d in zip(src, dst, data)]


@pytest.mark.parametrize("n,rk,dtype", [(24, 2, torch.float64), (90, 3, torch.float64), (136, 2, torch.float32)])
def test_phase_after_the_table_kernel_waits_for_it(n, rk, dtype, grids):
    g = grids(n)
    plan = BtPlan(make_consts(g, 5000.0), dtype=dtype)
    s = harmonic_state(g, 4)
    ins = [torch.from_numpy(np.ascontiguousarray(s[k])).to("cuda", dtype) for k in ("h0", "h0", "ub", "vb", "ub", "vb")]
    out = {k: plan.empty_field() for k in ("h0", "ub", "vb")}
    desc = N.GridDesc(n, N.BT_F64 if dtype == torch.float64 else N.BT_F32,
                      *[plan.consts[k].data_ptr() for k in CONST_NAMES])
    sin = N.StateIn(*[t.data_ptr() for t in ins])
    sout = N.StateOut(*[out[k].data_ptr() for k in ("h0", "ub", "vb")], (ctypes.c_void_p * 10)())
    stream = torch.cuda.Stream()

    def go(nbb):
        N.check(N.lib().bt_round_noalloc(ctypes.byref(desc), ctypes.byref(sin), ctypes.byref(sout), nbb, 10.0, rk,
                                         ctypes.c_void_p(stream.cuda_stream)))

    go(1)  # set-up and table check, outside a capture
    stream.synchronize()
    nbb = 3
    edges = _captured_edges(stream, lambda: go(nbb))
    # a chain: table kernel, 2 rk phases per substep, halo fill
    after = {a: (b, t) for a, b, t in edges}
    assert len(after) == len(edges) == 2 * rk * nbb + 1
    node = (set(after) - {b for _, b, _ in edges}).pop()
    kinds = []
    while node in after:
        node, kind = after[node]
        kinds.append(kind)
    assert kinds[0] == FULL
    assert set(kinds[1:2 * rk * nbb]) == {PROGRAMMATIC}
    plan.close()
