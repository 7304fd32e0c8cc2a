"""Batched double spherical-Bessel integrals on the GPU against the oracle (adaptive
Gauss-Legendre to 1e-14 on the same breakpoints) and the reference's own known values
(besseltools_test.py:26-58)."""
import numpy as np
import pytest

import catana_gb300 as catana
from catana_gb300 import besseltools
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def test_known_values(cuda_device):
    w = lambda r: np.ones_like(r)
    assert besseltools.double_sbessel_integrator(w, 0, 100, 1, 1) == pytest.approx(1.56582, abs=1e-5)
    assert besseltools.double_sbessel_integrator(w, 0, 100, 1, 2) == pytest.approx(0.785393, abs=1e-5)
    assert besseltools.double_sbessel_integrator(w, 4, 100, 1, 4.2) == pytest.approx(0.000133933, abs=1e-9)


def test_symmetric_and_interpolator(cuda_device):
    w = lambda r: np.exp(-(r / 40) ** 2) * r ** 2
    r1 = besseltools.double_sbessel_integrator(w, 6, 100, 2.3, 4.5)
    r2 = besseltools.double_sbessel_integrator(w, 6, 100, 4.5, 2.3)
    assert r1 == r2
    fi = catana.FunctionInterpolator(w, 100000, 0, 100)
    assert besseltools.double_sbessel_integrator(fi, 6, 100, 2.3, 4.5) == pytest.approx(r1, rel=1e-5)


@pytest.mark.parametrize("l,rmax,nodes,nk", [(0, 100.0, 20001, 6), (6, 100.0, 20001, 6), (20, 1000.0, 8001, 5),
                                          (100, 1000.0, 4001, 4)])
def test_vs_oracle(cuda_device, l, rmax, nodes, nk):
    """A batch of (k1, k2) pairs: zeros-of-j_l wave numbers as in a C_l^SN matrix."""
    fi = catana.FunctionInterpolator(lambda r: np.exp(-(r / (0.4 * rmax)) ** 2) * r ** 2, nodes, 0.0, rmax)
    k = catana.compute_kln(l + 1, nk, rmax)[l]
    k1, k2 = np.meshgrid(k, k)
    got = besseltools.double_sbessel_integrator(fi, l, rmax, k1, k2)
    scale = np.max(np.abs(got))
    for i in range(nk):
        for j in range(nk):
            ref = O.dsb_integral(fi.y_values, (fi.x_min, fi.x_max), l, rmax, k1[i, j], k2[i, j])
            assert abs(got[i, j] - ref) <= 1e-10 * scale, (i, j, got[i, j], ref)


@pytest.mark.parametrize("l,rmax,wmin,wmax,nodes", [(3, 100.0, 0.0, 100.0, 2), (3, 100.0, 0.0, 100.0, 7), (0, 37.3, -5.0, 60.0, 131),
                                                  (12, 50.0, -1.0, 50.0, 1001), (0, 10.0, 0.0, 12.0, 4001)])
def test_shared_quadrature_rules(cuda_device, l, rmax, wmin, wmax, nodes):
    """Every rule of the shared quadrature: segments cut into pieces (few nodes), 8, 4, 3 and 2 points, a table
    that reaches beyond [0, r_max) on both sides, k = 0 and equal k.  The rule errs below 1e-14, the oracle
    is adaptive to 1e-13, j_l carries ~1e-14: 1e-12 of the largest integral."""
    fi = catana.FunctionInterpolator(lambda r: 1.0 + np.cos(0.05 * r) * r, nodes, wmin, wmax)
    k = np.array([0.0, 1.0, 1.0]) * (30.0 if nodes < 1000 else 3.0 + l) / rmax
    k1, k2 = np.meshgrid(k, k)
    got = besseltools.double_sbessel_integrator(fi, l, rmax, k1, k2)
    ref = np.array([[O.dsb_integral(fi.y_values, (fi.x_min, fi.x_max), l, rmax, a, b) for a, b in zip(p, q)]
                    for p, q in zip(k1, k2)])
    assert np.max(np.abs(got - ref)) <= 1e-12 * np.max(np.abs(ref))


def test_many_distinct_k_in_passes(cuda_device):
    """4000 distinct k: the Bessel rows exceed one pass, the pairs' sums run over several."""
    rng = np.random.default_rng(2)
    fi = catana.FunctionInterpolator(lambda r: np.exp(-(r / 30) ** 2), 12001, 0.0, 100.0)
    k1, k2 = rng.uniform(0.05, 2.0, 2000), rng.uniform(0.05, 2.0, 2000)
    got = besseltools.double_sbessel_integrator(fi, 5, 100.0, k1, k2)
    one = np.array([besseltools.double_sbessel_integrator(fi, 5, 100.0, a, b) for a, b in zip(k1[:20], k2[:20])])
    assert np.max(np.abs(got[:20] - one)) <= 1e-13 * np.max(np.abs(one))


def test_one_large_k_does_not_set_the_others_rule(cuda_device):
    """200 pairs of small k and one whose segments take some 200 pieces each: two rules, a pass each (by one rule 3.2M nodes
    for 402 wave numbers, 41 passes), and each pair as by itself."""
    from catana_gb300 import _lib
    rng = np.random.default_rng(3)
    fi = catana.FunctionInterpolator(lambda r: np.exp(-(r / 30) ** 2), 2001, 0.0, 100.0)
    k1, k2 = rng.uniform(0.05, 2.0, 201), rng.uniform(0.05, 2.0, 201)
    k1[77], k2[77] = 6400.0, 6000.0
    n0 = _lib.lib.catana_gpu_launch_count()
    got = besseltools.double_sbessel_integrator(fi, 3, 100.0, k1, k2)
    assert _lib.lib.catana_gpu_launch_count() - n0 <= 6
    one = np.array([besseltools.double_sbessel_integrator(fi, 3, 100.0, a, b) for a, b in zip(k1, k2)])
    rest = np.arange(201) != 77
    assert np.max(np.abs(got - one)[rest]) <= 1e-13 * np.max(np.abs(one[rest]))
    assert abs(got[77] - one[77]) <= 1e-13 * abs(one[77])


def test_distinct_k_beyond_a_pass_memory(cuda_device):
    """100k distinct k: runs of pairs under 512 MB of Bessel rows (1.6 GB by one)."""
    from catana_gb300 import _lib
    rng = np.random.default_rng(4)
    fi = catana.FunctionInterpolator(lambda r: np.exp(-(r / 30) ** 2), 401, 0.0, 100.0)
    k1, k2 = rng.uniform(0.05, 2.0, 50000), rng.uniform(0.05, 2.0, 50000)
    _lib.lib.catana_gpu_test_alloc_limit(600 << 20)
    try:
        got = besseltools.double_sbessel_integrator(fi, 2, 100.0, k1, k2)
    finally:
        _lib.lib.catana_gpu_test_alloc_limit(0)
    some = np.concatenate([np.arange(0, 50000, 2500), [15624, 15625, 49999]])
    one = np.array([besseltools.double_sbessel_integrator(fi, 2, 100.0, k1[i], k2[i]) for i in some])
    assert np.max(np.abs(got[some] - one)) <= 1e-13 * np.max(np.abs(one))


def test_wave_numbers_past_any_rule_are_refused(cuda_device):
    """Also where the pieces are past every integer: an error before anything is computed."""
    fi = catana.FunctionInterpolator(lambda r: 1.0 + 0.0 * r, 11, 0.0, 100.0)
    for k in (1e10, 1e300, 1.7e308):
        with pytest.raises(ValueError):
            besseltools.double_sbessel_integrator(fi, 0, 100.0, np.array([1.0, k]), np.array([1.0, 1.0]))
