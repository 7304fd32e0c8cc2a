"""The sums and schedules around the kernels, at their edges: slabs of the split form's levels
(k_split_reduce), the weight sum, mode norms (k_finish), and the pixel offsets of the binning.

Tolerances: the split form's documented ones (max |df| <= 1e-5 max|f|, rms(df) <= 2e-5 rms(f) per
l); FP64 sums of n terms n 2^-53 of the magnitudes (at most 1e-9 here); offsets are exact.
"""
import numpy as np
import pytest

import catana_gb300 as catana
from oracle import oracle as O
from conftest import uniform_ball

pytestmark = pytest.mark.gpu


# one tile; slabs that do not divide the tiles; a slab per SM and one more; two halves, the second
# of one order; orders that do not fill a group of 32
@pytest.mark.parametrize("n,lmax,nmax", [(1, 3, 1), (33, 3, 33), (152 * 32, 4, 31), (152 * 32 + 1, 4, 32),
                                         (20000, 140, 129)])
def test_split_level_schedule(cuda_device, n, lmax, nmax):
    if tuple(cuda_device) != (10, 3):
        pytest.skip("split form needs sm_103")
    pc = catana.PointContainer(uniform_ball(n, 1000.0, seed=n + nmax))
    a = catana.sfb_decomposition(pc, lmax, nmax, 1000.0, True, False, precision="split")
    b = catana.sfb_decomposition(pc, lmax, nmax, 1000.0, True, False, interpolation="off")
    top = max(np.abs(y).max() for y in b.f_lmn)
    for x, y in zip(a.f_lmn, b.f_lmn):
        assert np.abs(x - y).max() <= 1e-5 * top
        assert np.sqrt(np.mean(np.abs(x - y) ** 2)) <= 2e-5 * np.sqrt(np.mean(np.abs(y) ** 2)) + 1e-12 * top


# one chunk, one more than a chunk, more chunks than CTAs
@pytest.mark.parametrize("n", [1, 1023, 8192, 8193, 592 * 8192 + 5])
def test_weight_sum(cuda_device, n):
    pts = np.zeros((n, 3))
    pts[:, 0] = 500.0  # one radius: f_00n of all points is the weights' mean times one point's
    w = np.random.default_rng(n).uniform(0.5, 1.5, n)
    a = catana.sfb_decomposition(catana.PointContainer(pts), 1, 1, 1000.0, True, False, weights=w)
    b = catana.sfb_decomposition(catana.PointContainer(pts), 1, 1, 1000.0, True, False)
    assert np.allclose(a.f_lmn[0], b.f_lmn[0], rtol=1e-9, atol=0.0)


@pytest.mark.parametrize("lmax,nmax", [(1, 1), (2, 33), (9, 32), (70, 31)])
def test_mode_norms(cuda_device, lmax, nmax):
    pts = uniform_ball(500, 1000.0, seed=lmax)
    res = catana.sfb_decomposition(catana.PointContainer(pts), lmax, nmax, 1000.0, True, False)
    for l in range(lmax):
        p = np.abs(res.f_lmn[l]) ** 2
        c = (p[0] + 2.0 * p[1:].sum(axis=0)) / (2 * l + 1)
        assert np.allclose(res.c_ln[l], c, rtol=1e-12, atol=0.0)


# fewer points than pixels, more, one pixel taking all; more sort tiles than one round of the scan
@pytest.mark.parametrize("nside,n,spread", [(1, 1, True), (2, 7, True), (64, 5000, True), (4, 4097, False),
                                            (2, 64 * 4096 + 1, True)])
def test_bin_offsets(cuda_device, nside, n, spread):
    pts = uniform_ball(n, 1000.0, seed=nside + n)
    if not spread:
        pts[:, 1:] = pts[0, 1:]
    ppc = catana.PixelizedPointContainer(nside, catana.PointContainer(pts))
    offs, rs = O.bin_points(nside, pts)
    assert np.array_equal(ppc.offsets, offs)
    assert np.array_equal(ppc.r_sorted, rs)
