"""The plain form on the tensor cores where a catalog, another call or a failed allocation gets in its way."""
import numpy as np
import pytest

import catana_gb300 as catana
from catana_gb300 import _lib
from conftest import uniform_ball

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("column,bad", [(1, np.nan), (1, np.inf), (2, np.nan), (2, -np.inf)])
@pytest.mark.parametrize("interp", ["on", "off"])
def test_angles_that_are_not_finite_keep_the_modes_they_do_not_enter(cuda_device, column, bad, interp):
    """theta does not enter l = 0, phi not m = 0: those sums hold the point as if its angle were any other.

    The two catalogs differ in one point's angle, the products of these modes not at all; only the order of
    the sums is free (~1e-15 of the largest), so 1e-13."""
    pts = uniform_ball(40, 1000.0, seed=9)  # one point is a fortieth of the sum
    pts[17, column] = bad
    ref = pts.copy()
    ref[17, column] = 0.75
    args = (4, 3, 1000.0, True, False)
    a = catana.sfb_decomposition(catana.PointContainer(pts), *args, interpolation=interp)
    b = catana.sfb_decomposition(catana.PointContainer(ref), *args, interpolation=interp)
    for l, (f, g) in enumerate(zip(a.f_lmn, b.f_lmn)):
        for m in range(l + 1):
            if (l if column == 1 else m) > 0:
                assert np.all(np.isnan(f[m])), (l, m)
            elif column == 1 or l == 0:
                assert np.max(np.abs(f[m] - g[m])) <= 1e-13 * np.max(np.abs(g[m])), (l, m)
            else:  # m = 0 of l > 0: the point's own theta
                assert np.max(np.abs(f[m] - g[m])) <= 1e-13 * np.max(np.abs(g)), (l, m)


def _raw(**kw):
    pts = uniform_ball(3000, 1000.0, seed=5)
    return lambda: catana.sfb_decomposition(catana.PointContainer(pts), 12, 20, 1000.0, True, False, interpolation="on", **kw)


def _healpix(reverse):
    ppc = catana.PixelizedPointContainer(8, catana.PointContainer(uniform_ball(3000, 1000.0, seed=5)))
    if reverse:
        return lambda: catana.sfb_reverse(ppc, 12, 20, 1000.0, True, False, interpolated=True)
    return lambda: catana.sfb_decomposition(ppc, 12, 20, 1000.0, True, False)


def _accumulator():
    pts = uniform_ball(3000, 1000.0, seed=5)

    def call():
        with catana.SFBAccumulator(12, 20, 1000.0, precision="plain") as acc:
            acc.add(pts)
            return acc.finish()

    return call


def _batched():
    pts = uniform_ball(3000, 1000.0, seed=5)
    return lambda: catana.sfb_decomposition_batched([catana.PointContainer(pts)], 12, 20, 1000.0, verbose=False,
                                                    precision="plain")[0]


@pytest.mark.parametrize("make", [_raw, lambda: _healpix(False), lambda: _healpix(True), _accumulator, _batched],
                         ids=["raw", "healpix", "reverse", "accumulator", "batched"])
def test_a_wait_that_runs_out_is_an_error(cuda_device, make):
    """The hook withholds one hand-off of the tensor-core kernel and cuts its waits to 3 ms: the call says so
    instead of returning what the kernel left, and the same call again is as before."""
    if tuple(cuda_device) != (10, 3):
        pytest.skip("the tensor-core kernel needs sm_103")
    call = make()
    before = call()
    assert _lib.lib.catana_gpu_test_plain_stall(3000) == _lib.OK
    with pytest.raises(_lib.CatanaError, match="timed-out"):
        call()
    after = call()
    assert np.array_equal(before.c_ln, after.c_ln)


def test_stall_hook_validates_its_argument():
    assert _lib.lib.catana_gpu_test_plain_stall(0) == _lib.ERR_ARG
    assert _lib.lib.catana_gpu_test_plain_stall(2000000) == _lib.ERR_ARG
