"""The plain form on the tensor cores where a catalog, another call or a failed allocation gets in its way."""
import numpy as np
import pytest

import catana_gb300 as catana
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
