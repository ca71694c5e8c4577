"""Which rounds run the fused stage kernel (BT_INFO_FUSED_ROUND: bit 0 RK2, bit 1 RK3, bit 2 tiles of 12 x 16).

On a B200 (148 SMs): from N = 18 (two tiles along each axis, none thinner than 6
cells), float64 RK2 up to two tiles per SM (N = 96, 12 x 16 tiles from N = 73), RK3 up to
1.75 of the 12 x 16 tiles (N = 84), float32 up to six (N = 128).  Both sides of each limit.
"""
import numpy as np
import pytest
import torch

from licom4py_gpu_b200 import _native as N
from licom4py_gpu_b200.duogrid import make_consts
from licom4py_gpu_b200.plan import BtPlan

pytestmark = pytest.mark.gpu
RK2, RK3, WIDE = 1, 2, 4


def _bits(plan):
    return int(N.lib().bt_plan_get_info(plan._h, N.BT_INFO_FUSED_ROUND))


@pytest.mark.parametrize("dtype,n,want", [
    (torch.float64, 17, 0), (torch.float64, 18, RK2 | RK3), (torch.float64, 72, RK2 | RK3),
    (torch.float64, 73, RK2 | RK3 | WIDE), (torch.float64, 84, RK2 | RK3 | WIDE), (torch.float64, 85, RK2 | WIDE),
    (torch.float64, 96, RK2 | WIDE), (torch.float64, 97, 0),
    (torch.float32, 17, 0), (torch.float32, 18, RK2 | RK3), (torch.float32, 73, RK2 | RK3 | WIDE),
    (torch.float32, 96, RK2 | RK3 | WIDE), (torch.float32, 97, RK2 | RK3), (torch.float32, 128, RK2 | RK3),
    (torch.float32, 129, 0)])
def test_fused_by_size(dtype, n, want, grids):
    p = BtPlan(make_consts(grids(n), 5000.0), dtype=dtype, tile=(8, 16))
    for mode in ("stream", "graph"):
        p.set_mode(mode)
        assert _bits(p) == want, mode
        p.set_tile(16, 16)  # another shape, one of the phase builds, another mode: the phases
        assert _bits(p) & (RK2 | RK3) == 0
        p.set_tile(8, 16)
        for full in (False, True):
            p.set_full_tiles(full)
            assert _bits(p) & (RK2 | RK3) == 0
        p.set_full_tiles(None)
    for mode in ("persistent", "resident"):
        p.set_mode(mode)
        assert _bits(p) & (RK2 | RK3) == 0
    p.close()


def test_far_sources_decline_the_fused_kernel(grids):
    """A halo cell interpolated from cells further along the edge than the kernel's patches reach."""
    g = grids(48)
    near = BtPlan(make_consts(g, 5000.0), tile=(8, 16))
    assert _bits(near) == RK2 | RK3
    near.close()
    consts = list(make_consts(g, 5000.0))
    loc = consts[6].copy()
    loc[0, 20, 0] += 9  # W band of face 0
    consts[6] = loc
    far = BtPlan(consts, tile=(8, 16))
    assert _bits(far) == 0
    far.close()
