"""The sums and schedules around the kernels, at their edges: slabs of the split form's levels
(k_split_reduce), the weight sum, mode norms (k_finish), and the pixel offsets of the binning.

Tolerances: the split form's documented ones (max |df| <= 1e-5 max|f|, rms(df) <= 2e-5 rms(f) per
l); FP64 sums of n terms n 2^-53 of the magnitudes (at most 1e-9 here); offsets are exact.
"""
import numpy as np
import pytest

import catana_gb300 as catana
from catana_gb300 import _lib
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


def _pixels(nside, pts):
    """The FP64 form on the device."""
    pix = np.zeros(len(pts), dtype=np.int64)
    th, ph = np.ascontiguousarray(pts[:, 1]), np.ascontiguousarray(pts[:, 2])
    _lib.check(_lib.lib.catana_gpu_ang2pix_ring(nside, _lib.ptr(th), _lib.ptr(ph), len(pts), _lib.ptr(pix), None))
    return pix


# pixels by FP32 where that settles them: the smallest nside, ordinary ones, the largest it takes and one past
@pytest.mark.parametrize("nside", [1, 2, 64, 1024])
def test_pixels_settled_in_fp32(cuda_device, nside):
    n = 200000
    rng = np.random.default_rng(nside)
    pts = uniform_ball(n, 1000.0, seed=nside)
    k = n // 8
    pts[:k, 1] = np.arccos(np.clip(rng.integers(-3, 4, k) / 3.0 + rng.choice([0, 1e-9, -1e-7, 3e-6], k), -1, 1))
    pts[k:2 * k, 2] = (np.pi / 2) * rng.integers(-4, 9, k) / 2.0 ** rng.integers(0, 7, k)
    pts[2 * k:3 * k, 2] += rng.choice([-4 * np.pi, 2 * np.pi, 100.0], k)
    pix = _pixels(nside, pts)
    ppc = catana.PixelizedPointContainer(nside, catana.PointContainer(pts))
    assert np.array_equal(np.diff(ppc.offsets), np.bincount(pix, minlength=12 * nside * nside))
    assert np.array_equal(ppc.r_sorted, pts[np.argsort(pix, kind="stable"), 0])


@pytest.mark.parametrize("nside,cartesian,f32", [(4, True, True), (64, True, False), (64, False, True), (512, True, True),
                                                 (2048, True, False)])
def test_ingest_mask_settled_in_fp32(cuda_device, nside, cartesian, f32):
    n = 150000
    rng = np.random.default_rng(nside)
    pts = uniform_ball(n, 1000.0, seed=nside + 1)
    rec = pts
    if cartesian:
        st = np.sin(pts[:, 1])
        rec = pts[:, :1] * np.stack([st * np.cos(pts[:, 2]), st * np.sin(pts[:, 2]), np.cos(pts[:, 1])], 1)
        rec[:1000, rng.integers(0, 3)] = 0.0
        rec[1000:1100] *= 1e-25
        rec[0] = 0.0
    rec = rec.astype(np.float32) if f32 else np.ascontiguousarray(rec)
    mask = rng.integers(0, 2, 12 * nside * nside).astype(np.float32)
    kind = "cartesian" if cartesian else "spherical"
    got = np.asarray(catana.ingest(rec, kind, mask=mask, tophat_r0=900.0))
    ref = np.asarray(catana.ingest(rec, kind, tophat_r0=900.0))
    assert np.array_equal(got, ref[mask[_pixels(nside, ref)] == 1.0])
