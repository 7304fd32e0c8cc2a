"""The plain form's tensor-core contraction (k_ptc_main) at the sizes where its tiling can go wrong:
point counts around a tile (32), a group (128) and a slab, multipoles around the 64-row blocks, radial
orders around the 16-column steps, the 32-column halves and the 64-column blocks; weights that vary by
many orders; points that are not finite.

Tolerance, from the arithmetic: digits are cut at 2^-55 of a row's bound and sums at 2^-51 of a slab's
largest term, ~1e-15; the oracle's own table position k r / dx carries a rounding of 1e5 * 2^-53 in a slope of
~3e-3 (4e-14 of j_l's envelope), and both recurrences build up ~l 2^-53.  1e-12 of the level's largest
|f| leaves a factor of ten over their sum."""
import numpy as np
import pytest

import catana_gb300 as catana
from oracle import oracle as O
from conftest import uniform_ball

pytestmark = pytest.mark.gpu
TOL = 1e-12


def _check(pts, lmax, nmax, interp, weights=None, rmax=1000.0):
    res = catana.sfb_decomposition(catana.PointContainer(pts), lmax, nmax, rmax, True, False, weights=weights,
                                   interpolation=interp)
    k, c, f = O.sfb_raw(pts, lmax, nmax, rmax, interpolated=(interp == "on"), weights=weights)
    assert np.array_equal(res.k_ln, k)
    for l, (a, b) in enumerate(zip(res.f_lmn, f)):
        assert np.max(np.abs(a - b)) <= TOL * np.max(np.abs(b)), (l, np.max(np.abs(a - b)) / np.max(np.abs(b)))


@pytest.mark.parametrize("n,lmax,nmax", [(1, 1, 1), (31, 2, 16), (32, 5, 17), (33, 33, 32), (129, 64, 33), (300, 65, 48),
                                         (161, 66, 64), (700, 70, 65), (5000, 34, 130)])
def test_tile_edges(cuda_device, n, lmax, nmax):
    pts = uniform_ball(n, 1000.0, seed=n)
    _check(pts, lmax, nmax, "on")
    if n <= 200:
        _check(pts, lmax, nmax, "off")
        _check(pts, lmax, nmax, "poly", np.random.default_rng(1).uniform(0.5, 1.5, n))


def test_many_slabs_and_groups(cuda_device):
    """More than one slab per CTA slot is not needed here: 40k points give slabs of nine tiles, a last group
    of one tile, and sixteen-column D regions that alternate."""
    _check(uniform_ball(40000, 1000.0, seed=3), 7, 16, "on")


def test_narrow_catalogs(cuda_device):
    """Points in a polar cap and in a thin, distant shell: the row bounds follow the points (|P_lm| down to
    sin(0.05)^m, j_l far below its first maximum) and the small values keep their digits."""
    rng = np.random.default_rng(5)
    n = 400
    cap = np.stack([1000.0 * rng.random(n) ** (1 / 3), rng.uniform(0.01, 0.05, n), rng.uniform(0, 2 * np.pi, n)], 1)
    _check(cap, 24, 12, "on")
    near = cap.copy()
    near[:, 0] = rng.uniform(20.0, 25.0, n)
    near[:, 1] = np.arccos(rng.uniform(-1, 1, n))
    _check(near, 24, 12, "off")
    same = np.tile(np.array([[700.0, 1.1, 2.2]]), (n, 1))  # every digit the same: the sums' largest values
    _check(same, 24, 12, "on")


def test_weights_over_many_orders(cuda_device):
    rng = np.random.default_rng(6)
    pts = uniform_ball(3000, 1000.0, seed=8)
    _check(pts, 12, 20, "on", 10.0 ** rng.uniform(-9, 3, 3000))
    _check(pts, 12, 20, "on", rng.normal(size=3000))
    _check(pts, 12, 20, "on", np.where(np.arange(3000) == 17, 1.0, 0.0))


@pytest.mark.parametrize("column,bad", [(1, np.nan), (2, np.inf), (3, np.nan)])
def test_points_that_are_not_finite(cuda_device, column, bad):
    """theta enters every l > 0, phi every m > 0, a weight everything; the rest stays as without the flaw."""
    pts = uniform_ball(200, 1000.0, seed=9)
    w = np.ones(200)
    if column < 3:
        pts[50, column] = bad
    else:
        w[50] = bad
    res = catana.sfb_decomposition(catana.PointContainer(pts), 4, 3, 1000.0, True, False, weights=w, interpolation="on")
    for l, f in enumerate(res.f_lmn):
        for m in range(l + 1):
            nan = (column == 1 and l > 0) or (column == 2 and m > 0) or column == 3
            assert np.all(np.isnan(f[m])) == nan and np.all(np.isfinite(f[m])) == (not nan), (l, m)


@pytest.mark.parametrize("nside,n,lmax,nmax", [(1, 40, 12, 3), (2, 300, 20, 16), (8, 1500, 40, 33), (16, 30000, 8, 8), (4, 5000, 6, 5)])
@pytest.mark.parametrize("dense", [False, True])
def test_pixelized_points(cuda_device, nside, n, lmax, nmax, dense):
    """The pixelized sum point by point at pixel centres, polar rings shorter than 2 l included (aliases with
    and without the conjugate)."""
    pts = uniform_ball(n, 1000.0, seed=n + nside)
    ppc = catana.PixelizedPointContainer(nside, catana.PointContainer(pts))
    if dense:
        res = catana.sfb_reverse(ppc, lmax, nmax, 1000.0, True, False, interpolated=True)
        k, c, f = O.sfb_reverse(nside, ppc.offsets, ppc.r_sorted, lmax, nmax, 1000.0, interpolated=True)
    else:
        res = catana.sfb_decomposition(ppc, lmax, nmax, 1000.0, True, False, interpolation="on")
        k, c, f = O.sfb_healpix(nside, ppc.offsets, ppc.r_sorted, lmax, nmax, 1000.0, interpolated=True)
    for l, (a, b) in enumerate(zip(res.f_lmn, f)):
        assert np.max(np.abs(a - b)) <= TOL * max(np.max(np.abs(b)), 1e-6 * np.max(np.abs(f[0]))), l


@pytest.mark.parametrize("nside,counts", [(1, (64,)), (1, (65, 1)), (2, (129, 63, 64, 1)), (2, (3000,)), (4, (1,) * 33 + (200,))])
@pytest.mark.parametrize("interpolated", [True, False])
def test_pixelized_cells(cuda_device, nside, counts, interpolated):
    """Pixels with less, just as many and more points than are summed at once; entries of unlike counts in a tile."""
    npix = 12 * nside * nside
    offs = np.zeros(npix + 1, dtype=np.int64)
    offs[1:] = np.cumsum(np.bincount((7 * np.arange(len(counts)) + 3) % npix, weights=counts, minlength=npix))
    n = int(offs[-1])
    r = 1000.0 * np.random.default_rng(n).uniform(0.0, 1.0, n) ** (1.0 / 3.0)
    ppc = catana.PixelizedPointContainer(nside)
    ppc.offsets, ppc.r_sorted = offs, r
    res = catana.sfb_decomposition(ppc, 9, 11, 1000.0, True, False, interpolation="on" if interpolated else "off")
    k, c, f = O.sfb_healpix(nside, offs, r, 9, 11, 1000.0, interpolated=interpolated)
    for l, (a, b) in enumerate(zip(res.f_lmn, f)):
        assert np.max(np.abs(a - b)) <= TOL * max(np.max(np.abs(b)), 1e-6 * np.max(np.abs(f[0]))), l


@pytest.mark.parametrize("n,lmax,nmax", [(1, 1, 1), (40, 2, 1), (500, 8, 64), (500, 8, 193), (2000, 4, 300), (8192, 1, 64), (8193, 1, 64),
                                         (100, 64, 200), (100, 65, 200)])
@pytest.mark.parametrize("interp", ["on", "off"])
def test_small_catalogs_either_path(cuda_device, n, lmax, nmax, interp):
    """Both sides of the rule that leaves few points with many radial orders to the FP64 path."""
    pts = uniform_ball(n, 1000.0, seed=n + nmax)
    res = catana.sfb_decomposition(catana.PointContainer(pts), lmax, nmax, 1000.0, True, False, interpolation=interp)
    keep = min(lmax, 6)  # the oracle's levels
    k, c, f = O.sfb_raw(pts, keep, nmax, 1000.0, interpolated=interp == "on")
    for l in range(keep):
        assert np.max(np.abs(res.f_lmn[l] - f[l])) <= 1e-10 * max(np.max(np.abs(f[0])), np.max(np.abs(f[l])))
