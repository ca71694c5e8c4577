"""Every form of a float32 round gives the same bits.

Float32 keeps fused multiply-adds, and each sum that takes part in one names the
product that is fused, so the phase kernels of every tile shape and build, the
fused stage kernel, the persistent and resident rounds and the batches compute
the same state to the bit.
"""
import numpy as np
import pytest
import torch

from licom4py_gpu_b200 import _native as N
from licom4py_gpu_b200.batch import BtBatch, MemberState
from licom4py_gpu_b200.duogrid import make_consts
from licom4py_gpu_b200.fields import cfl_dtb, harmonic_state
from licom4py_gpu_b200.plan import BtPlan

pytestmark = pytest.mark.gpu
F32 = torch.float32
TILES = [(8, 16), (8, 32), (16, 16), (16, 32), (7, 32), (15, 32)]


def _setup(g, n):
    s, b = harmonic_state(g, n), harmonic_state(g, n + 20, 0.5, 0.1)
    ins = [torch.from_numpy(np.ascontiguousarray(a)).to("cuda", F32)
           for a in (s["h0"], b["h0"], s["ub"], s["vb"], b["ub"], b["vb"])]
    return make_consts(g, 5000.0), ins, cfl_dtb(g, 5000.0)


def _same(want, got, what):
    for k in ("h0", "ub", "vb"):
        assert torch.equal(want[k], got[k]), (what, k)


@pytest.mark.parametrize("rk", [2, 3])
@pytest.mark.parametrize("n", [17, 24, 33, 48, 72, 77, 96, 128, 129])
def test_plan_forms_give_the_same_bits(n, rk, grids):
    consts, ins, dtb = _setup(grids(n), n)
    kw = dict(nbb=5, dtb=dtb, rk=rk, diag=False)
    p = BtPlan(consts, dtype=F32, tile=(8, 16))
    fused = int(N.lib().bt_plan_get_info(p._h, N.BT_INFO_FUSED_ROUND)) & 3
    assert fused == (3 if 17 < n <= 128 else 0)
    want = p.round(*ins, **kw)
    for tile in TILES:
        p.set_tile(*tile)
        for full in (False, True):
            p.set_full_tiles(full)
            _same(want, p.round(*ins, **kw), (tile, full))
        p.set_full_tiles(None)
        p.set_mode("persistent")
        _same(want, p.round(*ins, **kw), (tile, "persistent"))
        if tile in ((8, 16), (16, 16), (8, 32)) and n <= 96:
            p.set_mode("resident")
            _same(want, p.round(*ins, **kw), (tile, "resident"))
        p.set_mode("stream")
        p.check_device_error()
    p.close()


@pytest.mark.parametrize("mode", ["stream", "persistent"])
@pytest.mark.parametrize("tile", TILES)
def test_batches_give_the_bits_of_a_plan(mode, tile, grids):
    plans, members, want = {}, [], []
    for n in (24, 48, 96):
        consts, ins, dtb = _setup(grids(n), n)
        plans[n] = BtPlan(consts, dtype=F32, tile=(8, 16))
        h, u, v = ins[0], ins[2], ins[3]
        want.append(plans[n].round(h, h, u, v, u, v, nbb=6, dtb=dtb, diag=False))
        members.append(MemberState(plans[n], h, u, v, 6, dtb))
    b = BtBatch(F32, max_members=4, mode=mode, tile=tile)
    b.advance(members)
    for m, w in zip(members, want):
        for k, t in zip(("h0", "ub", "vb"), m.state):
            assert torch.equal(w[k], t), (m.plan.n, k)
    for p in plans.values():
        p.close()
