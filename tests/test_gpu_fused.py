"""Fused stage kernel (phase UV of a stage and phase H of the next in one launch).

It computes each value with the phase kernels' own expressions, so float64
rounds must equal the phases' (``set_full_tiles`` forces them) bit for bit;
float32 is held to 1e-6 relative (max norm), as other forms of the same round,
whose contraction choices may differ.  Sizes: the smallest it takes, face
extents that 8 x 16 does and does not divide, uneven splits, more than one tile
per SM, sizes where it takes 12 x 16 tiles, and a size below its range.
"""
import numpy as np
import pytest
import torch

from helpers import rel_err
from licom4py_gpu_b200.duogrid import make_consts
from licom4py_gpu_b200.fields import cfl_dtb, harmonic_state
from licom4py_gpu_b200.plan import BtPlan

pytestmark = pytest.mark.gpu


def inputs(g, seed, dtype):
    s, b = harmonic_state(g, seed), harmonic_state(g, seed + 20, 0.5, 0.1)
    return [torch.from_numpy(np.ascontiguousarray(a)).to("cuda", dtype)
            for a in (s["h0"], b["h0"], s["ub"], s["vb"], b["ub"], b["vb"])]


@pytest.mark.parametrize("n", [17, 18, 25, 33, 41, 48, 58, 72, 77, 84, 96])
@pytest.mark.parametrize("rk", [2, 3])
def test_fused_round_bitwise_equals_phases_f64(n, rk, grids):
    g = grids(n)
    consts = make_consts(g, 5000.0)
    ins = inputs(g, n, torch.float64)
    dtb = cfl_dtb(g, 5000.0)
    ref = BtPlan(consts, tile=(8, 16))
    ref.set_full_tiles(False)
    for nbb in (1, 2, 5):
        want = ref.round(*ins, nbb=nbb, dtb=dtb, rk=rk)
        for mode in ("stream", "graph"):
            p = BtPlan(consts, tile=(8, 16), mode=mode)
            for _ in range(2):
                got = p.round(*ins, nbb=nbb, dtb=dtb, rk=rk)
                for k in want:
                    assert torch.equal(want[k], got[k]), (n, rk, nbb, mode, k)
            p.close()
    ref.close()


@pytest.mark.parametrize("n,rk", [(18, 2), (48, 3), (90, 2), (96, 3), (112, 3)])
def test_fused_round_matches_phases_f32(n, rk, grids):
    g = grids(n)
    consts = make_consts(g, 5000.0)
    ins = inputs(g, n, torch.float32)
    dtb = cfl_dtb(g, 5000.0)
    p = BtPlan(consts, dtype=torch.float32, tile=(8, 16))
    got = p.round(*ins, nbb=5, dtb=dtb, rk=rk)
    p.set_full_tiles(False)
    want = p.round(*ins, nbb=5, dtb=dtb, rk=rk)
    for k in ("h0", "ub", "vb"):
        assert rel_err(got[k].cpu(), want[k].cpu()) <= 1e-6, (n, rk, k)
    p.close()


def test_tables_with_far_sources_keep_the_phases(grids):
    """A halo cell interpolated from cells further along the edge than the fused kernel's patches
    reach: the plan must not use it."""
    g = grids(48)
    consts = list(make_consts(g, 5000.0))
    loc = consts[6].copy()
    loc[0, 20, 0] += 9  # W band of face 0
    consts[6] = loc
    ins = inputs(g, 5, torch.float64)
    p = BtPlan(consts, tile=(8, 16))
    got = p.round(*ins, nbb=3, dtb=10.0)
    p.set_full_tiles(False)
    want = p.round(*ins, nbb=3, dtb=10.0)
    for k in want:
        assert torch.equal(want[k], got[k]), k
    p.close()
