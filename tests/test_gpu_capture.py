"""Rounds captured by the caller on its own stream.

The first stage or round of a plan with its tile shape prepares everything a
round needs, whatever entry point and options it runs with; from then on a
stream-mode round only launches kernels and can be captured and replayed.
"""
import numpy as np
import pytest
import torch

from licom4py_gpu_b200.duogrid import make_consts
from licom4py_gpu_b200.fields import cfl_dtb, harmonic_state
from licom4py_gpu_b200.plan import BtPlan

pytestmark = pytest.mark.gpu


def _inputs(g, seed):
    s, b = harmonic_state(g, seed), harmonic_state(g, seed + 20, 0.5, 0.1)
    return [torch.from_numpy(np.ascontiguousarray(a)).cuda()
            for a in (s["h0"], b["h0"], s["ub"], s["vb"], b["ub"], b["vb"])]


# C90 float64: RK2 rounds run the fused stage kernel, RK3 rounds the phase kernels; C24: both fused
@pytest.mark.parametrize("n,warm", [(24, "stage"), (24, "phases"), (24, "timed"), (24, "rk3"), (90, "rk3"),
                                    (90, "stage"), (17, "stage")])
def test_round_in_the_callers_capture(n, warm, grids):
    g = grids(n)
    consts = make_consts(g, 5000.0)
    ins = _inputs(g, n)
    dtb = cfl_dtb(g, 5000.0)
    ref = BtPlan(consts, tile=(8, 16))
    want = ref.round(*ins, nbb=3, dtb=dtb)
    p = BtPlan(consts, tile=(8, 16))
    if warm == "stage":
        p.stage(*ins, dt=dtb, beta_d=0.0, is_laststep=True)
    elif warm == "rk3":
        p.round(*ins, nbb=1, dtb=dtb, rk=3)
    elif warm == "phases":
        p.set_full_tiles(False)
        p.round(*ins, nbb=1, dtb=dtb)
        p.set_full_tiles(None)
    else:
        p.enable_kernel_timing(True)
        p.round(*ins, nbb=1, dtb=dtb)
        p.enable_kernel_timing(False)
    out = {k: p.empty_field() for k in want}
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        p.round(*ins, nbb=3, dtb=dtb, out=out)
    for _ in range(2):
        for t in out.values():
            t.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for k in want:
            assert torch.equal(want[k], out[k]), (n, warm, k)
    graph.reset()
    p.close()
    ref.close()
