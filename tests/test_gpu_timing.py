"""Kernel timing (BT_OPT_KERNEL_TIMING) and the kernels a round runs.

Stream mode times each phase kernel, so a round that would run the fused stage
kernel runs the phases while timing is on.  A graph round is not timed: what it
runs does not depend on the option, before or after it was captured.
"""
import numpy as np
import pytest
import torch

from licom4py_gpu_b200 import _native as N
from licom4py_gpu_b200.duogrid import make_consts
from licom4py_gpu_b200.fields import cfl_dtb, harmonic_state
from licom4py_gpu_b200.plan import BtPlan

pytestmark = pytest.mark.gpu


def _fused(plan):
    return int(N.lib().bt_plan_get_info(plan._h, N.BT_INFO_FUSED_ROUND)) & 3


def _setup(g, mode, tile=(8, 16)):
    s = harmonic_state(g, 3)
    ins = [torch.from_numpy(np.ascontiguousarray(s[k])).cuda() for k in ("h0", "h0", "ub", "vb", "ub", "vb")]
    return BtPlan(make_consts(g, 5000.0), tile=tile, mode=mode), ins, cfl_dtb(g, 5000.0)


def test_stream_timing_runs_and_counts_the_phases(grids):
    p, ins, dtb = _setup(grids(24), "stream")
    assert _fused(p) == 3
    want = p.round(*ins, nbb=4, dtb=dtb)
    p.enable_kernel_timing(True)
    assert _fused(p) == 0
    got = p.round(*ins, nbb=4, dtb=dtb)
    assert p.kernel_time("phase_h")[1] == p.kernel_time("phase_uv")[1] == 8
    p.enable_kernel_timing(False)
    assert _fused(p) == 3
    for k in want:
        assert torch.equal(want[k], got[k]), k
    p.close()


@pytest.mark.parametrize("tile", [(8, 16), (16, 16)])  # fused, phases
@pytest.mark.parametrize("first", [False, True])
def test_graph_rounds_are_the_same_with_timing_on_or_off(tile, first, grids):
    p, ins, dtb = _setup(grids(24), "graph", tile)
    fused = _fused(p)
    assert fused == (3 if tile == (8, 16) else 0)
    want = None
    for on in (first, not first, first):  # the first round is captured, the others replay it
        p.enable_kernel_timing(on)
        assert _fused(p) == fused
        got = p.round(*ins, nbb=4, dtb=dtb)
        for kind in ("phase_h", "phase_uv"):
            assert p.kernel_time(kind) == (0.0, 0)
        want = want or {k: v.clone() for k, v in got.items()}
        for k in want:
            assert torch.equal(want[k], got[k]), (on, k)
    p.close()
