"""Interior statistics and conservation sums against exactly rounded sums on the host.

Sizes around the kernels' column strips (192 and 96), the smallest, and one
with several strips per warp.  The sums are compensated: what is left is the
rounding of the compensation and of the final sum and quotient, at most
4 x 2^-53 of the result (plus 1e-20 of the mean magnitude for the second-order
terms).  Maximum and minimum are exact.
"""
import math

import numpy as np
import pytest
import torch

from licom4py_gpu_b200.momentum import conservation, interior_stats

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


@pytest.mark.parametrize("n", [1, 5, 31, 95, 96, 97, 191, 192, 193, 256])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_reductions_match_exact_sums(n, dtype):
    rng = np.random.default_rng(n)
    m = n + 6
    npt = np.float64 if dtype == torch.float64 else np.float32
    h, u, v = (rng.standard_normal((6, m, m)).astype(npt) for _ in range(3))
    rda = (1e-10 * (1.0 + rng.random((6, m, m)))).astype(npt)
    c2l = rng.standard_normal((6, m, m, 2, 2)).astype(npt)
    dev = [torch.from_numpy(a).cuda() for a in (h, u, v, rda, c2l)]
    inside = (slice(None), slice(3, -3), slice(3, -3))
    x = h[inside].astype(np.float64).ravel()
    got = interior_stats(dev[0]).cpu().numpy()
    assert got[0] == x.max() and got[1] == x.min()
    want = math.fsum(x) / x.size
    assert abs(got[2] - want) <= 4 * EPS * abs(want) + 1e-20 * np.abs(x).mean()
    if dtype == torch.float64:  # the terms' expressions round alike without FMA contraction
        hi, ui, vi, ri, c = (a[inside] for a in (h, u, v, rda, c2l))
        da = 1.0 / ri
        ul = c[..., 0, 0] * ui + c[..., 0, 1] * vi
        vl = c[..., 1, 0] * ui + c[..., 1, 1] * vi
        mass = (hi * da).ravel()
        energy = ((0.5 * 9.8 * hi * hi + 0.5 * (5000.0 + hi) * (ul * ul + vl * vl)) * da).ravel()
        got = conservation(*dev, 5000.0).cpu().numpy()
        for g, t in zip(got, (mass, energy)):
            want = math.fsum(t)
            assert abs(g - want) <= 4 * EPS * abs(want) + 1e-20 * np.abs(t).sum()


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_conservation_of_matrices_off_a_16_byte_boundary(dtype):
    """Matrices that start off a 16-byte boundary are read one value at a time: the same sums to the bit."""
    gen = torch.Generator().manual_seed(3)
    f = [torch.rand((6, 39, 39), generator=gen, dtype=torch.float64).to("cuda", dtype) + 0.5 for _ in range(4)]
    c = torch.randn((6 * 39 * 39 * 4 + 1,), generator=gen, dtype=torch.float64).to("cuda", dtype)
    off = c[1:].view(6, 39, 39, 2, 2)
    assert off.data_ptr() % 16 != 0 and off.clone().data_ptr() % 16 == 0
    assert torch.equal(conservation(*f, off, 5000.0), conservation(*f, off.clone(), 5000.0))
