"""The paths that sizes past the tensor-core kernel's take (lmax > 512): the FP64 kernels of the raw sum, and the maps, ring
transforms and folded sums of the pixelized one -- at every level against the tensor-core kernel, which shares
none of their code, and at the lowest against the oracle; and the tensor-core kernel's sums at their fullest.

Tolerance: the two sides differ by the table position's rounding (1e5 * 2^-53 in a slope of ~3e-3: 4e-14 of j_l's
envelope) and by recurrences over l <= 512 (~l 2^-53: 6e-14); 1e-11 of a level's largest |f| leaves a factor of a
hundred, 1e-10 of the largest |f| is the bar of the other pixelized tests against the oracle."""
import numpy as np
import pytest

import catana_gb300 as catana
from oracle import oracle as O
from conftest import uniform_ball

pytestmark = pytest.mark.gpu


def _sum(ppc, lmax, nmax, interp, dense):
    if dense:
        return catana.sfb_reverse(ppc, lmax, nmax, 1000.0, True, False, interpolated=interp)
    return catana.sfb_decomposition(ppc, lmax, nmax, 1000.0, True, False, interpolation="on" if interp else "off")


@pytest.mark.parametrize("nside,n,lmax,nmax,keep", [(1, 40, 513, 2, 513),  # every ring has 4 pixels
                                                    (8, 300, 516, 3, 40),   # rings of 4 to 32 pixels
                                                    (32, 2000, 520, 1, 30),  # 128 pixels: the FFT from l = 24 on
                                                    (64, 300, 514, 2, 40)])  # 256 pixels: from l = 28 on
@pytest.mark.parametrize("interp", [True, False])
@pytest.mark.parametrize("dense", [False, True])
def test_maps_and_ring_transforms(cuda_device, nside, n, lmax, nmax, keep, interp, dense):
    ppc = catana.PixelizedPointContainer(nside, catana.PointContainer(uniform_ball(n, 1000.0, seed=nside)))
    res = _sum(ppc, lmax, nmax, interp, dense)
    # polar rings of few pixels alias, so a level holds sums far above its points' own harmonics: one scale for all
    fmax = max(np.max(np.abs(f)) for f in res.f_lmn)
    tc = _sum(ppc, 512, nmax, interp, dense)
    for l in range(512):
        assert np.max(np.abs(res.f_lmn[l] - tc.f_lmn[l])) <= 1e-10 * fmax, l
    oracle = O.sfb_reverse if dense else O.sfb_healpix
    k, c, f = oracle(nside, ppc.offsets, ppc.r_sorted, keep, nmax, 1000.0, interpolated=interp)
    assert np.array_equal(res.k_ln[:keep], k)
    for l in range(keep):
        assert np.max(np.abs(res.f_lmn[l] - f[l])) <= 1e-10 * fmax, l


@pytest.mark.parametrize("n,lmax,nmax,interp", [(9000, 513, 2, "on"), (9000, 514, 2, "poly"), (20000, 513, 3, "off")])
def test_fp64_kernels(cuda_device, n, lmax, nmax, interp):
    pts = uniform_ball(n, 1000.0, seed=n)
    w = np.random.default_rng(n).uniform(0.5, 1.5, n)

    def call(lmax):
        return catana.sfb_decomposition(catana.PointContainer(pts), lmax, nmax, 1000.0, True, False, weights=w,
                                        interpolation=interp).f_lmn

    res, tc = call(lmax), call(512)
    for l in range(512):
        assert np.max(np.abs(res[l] - tc[l])) <= 1e-11 * np.max(np.abs(tc[l])), l
    f = O.sfb_raw(pts, 6, nmax, 1000.0, interpolated=interp == "on", weights=w)[2]
    for l in range(6):
        assert np.max(np.abs(res[l] - f[l])) <= 1e-10 * np.max(np.abs(f[l])), l


@pytest.mark.parametrize("nmax", [16, 48])
def test_the_largest_sums_of_a_slab(cuda_device, nmax):
    """Identical points in full slabs (64 tiles, 16 groups of 128): every FP32 sum of digits, every group's sum and the counts
    above 2^60 reach what they can; with 48 radial orders in both column regions.  The mean over the catalog is the point's
    own value: 1e-12."""
    n = 152 * 64 * 32
    point = np.array([[612.5, 1.1, 2.2]])

    def call(pts):
        return catana.sfb_decomposition(catana.PointContainer(pts), 4, nmax, 1000.0, True, False, interpolation="on").f_lmn

    many, one = call(np.tile(point, (n, 1))), call(np.tile(point, (33, 1)))
    for l in range(4):
        assert np.max(np.abs(many[l] - one[l])) <= 1e-12 * np.max(np.abs(one[l])), l


def test_several_groups_in_both_column_regions(cuda_device):
    """Six tiles a slab with 48 radial orders, against the oracle."""
    pts = uniform_ball(152 * 32 * 6, 1000.0, seed=3)
    res = catana.sfb_decomposition(catana.PointContainer(pts), 5, 48, 1000.0, True, False, interpolation="on")
    f = O.sfb_raw(pts, 5, 48, 1000.0, interpolated=True)[2]
    for l in range(5):
        assert np.max(np.abs(res.f_lmn[l] - f[l])) <= 1e-12 * np.max(np.abs(f[l])), l
