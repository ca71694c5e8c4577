"""The reductions on every cluster size, down to the single CTA that runs where no cluster can be placed.

Against exactly rounded sums on the host, with the bound of the compensated sums
(4 x 2^-53 of the result, plus 1e-20 of the mean magnitude for the second-order
terms), which does not depend on the order in which they are combined.
"""
import ctypes
import math

import numpy as np
import pytest
import torch

from licom4py_gpu_b200 import _native as N
from licom4py_gpu_b200.momentum import conservation, interior_stats

EPS = 2.0 ** -53


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def _stats(ctas, field):
    out = torch.empty(3, dtype=torch.float64, device="cuda")
    N.check(N.lib().bt_interior_stats_on(ctas, field.shape[-1] - 6, N.BT_F64, _ptr(field), _ptr(out),
                                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return out.cpu().numpy()


def _conservation(ctas, fields, depth):
    out = torch.empty(2, dtype=torch.float64, device="cuda")
    N.check(N.lib().bt_conservation_on(ctas, fields[0].shape[-1] - 6, N.BT_F64, *[_ptr(t) for t in fields], depth,
                                       _ptr(out), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return out.cpu().numpy()


@pytest.mark.parametrize("ctas", [-1, 3, 12, 17, 32])
def test_other_cta_counts_are_refused(ctas):
    lib = N.lib()
    p = ctypes.c_void_p(0x10000)  # never dereferenced: the argument checks come first
    assert lib.bt_interior_stats_on(ctas, 8, N.BT_F64, p, p, None) == N.BT_EINVAL
    assert lib.bt_conservation_on(ctas, 8, N.BT_F64, p, p, p, p, p, 1.0, p, None) == N.BT_EINVAL


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 33, 97, 193])
def test_every_cluster_size_gives_the_sums(n):
    rng = np.random.default_rng(n)
    m = n + 6
    h, u, v = (rng.standard_normal((6, m, m)) for _ in range(3))
    rda = 1e-10 * (1.0 + rng.random((6, m, m)))
    c2l = rng.standard_normal((6, m, m, 2, 2))
    dev = [torch.from_numpy(a).cuda() for a in (h, u, v, rda, c2l)]
    inside = (slice(None), slice(3, -3), slice(3, -3))
    x = h[inside].ravel()
    hi, ui, vi, ri, c = (a[inside] for a in (h, u, v, rda, c2l))
    da = 1.0 / ri
    ul = c[..., 0, 0] * ui + c[..., 0, 1] * vi
    vl = c[..., 1, 0] * ui + c[..., 1, 1] * vi
    terms = ((hi * da).ravel(),
             ((0.5 * 9.8 * hi * hi + 0.5 * (5000.0 + hi) * (ul * ul + vl * vl)) * da).ravel())
    for ctas in (1, 2, 4, 8, 16):
        got = _stats(ctas, dev[0])
        assert got[0] == x.max() and got[1] == x.min()
        want = math.fsum(x) / x.size
        assert abs(got[2] - want) <= 4 * EPS * abs(want) + 1e-20 * np.abs(x).mean(), ctas
        for g, t in zip(_conservation(ctas, dev, 5000.0), terms):
            want = math.fsum(t)
            assert abs(g - want) <= 4 * EPS * abs(want) + 1e-20 * np.abs(t).sum(), ctas
    # a whole GPU runs the 16
    assert np.array_equal(interior_stats(dev[0]).cpu().numpy(), _stats(16, dev[0]))
    assert np.array_equal(conservation(*dev, 5000.0).cpu().numpy(), _conservation(16, dev, 5000.0))


@pytest.mark.gpu
@pytest.mark.parametrize("bad", [math.nan, math.inf, -math.inf])
def test_one_cta_and_the_cluster_treat_non_finite_cells_alike(bad):
    f = torch.randn(6, 39, 39, dtype=torch.float64, device="cuda")
    f[3, 20, 11] = bad
    assert np.array_equal(_stats(1, f), _stats(16, f), equal_nan=True)
