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


def _interleaved(shapes, chunks, interp):
    """Accumulators of unlike nmax fed in turn: each one's table replaces the others' in the shared cache."""
    accs = [catana.SFBAccumulator(lmax, nmax, rmax, precision="plain", interpolation=interp) for lmax, nmax, rmax in shapes]
    for c in chunks:
        for a in accs:
            a.add(c)
    out = [a.finish(store_flmn=True) for a in accs]
    for a in accs:
        a.close()
    return out


@pytest.mark.parametrize("interp,shapes", [("on", [(24, 64, 1000.0), (24, 32, 1000.0), (9, 48, 1000.0)]),
                                           ("poly", [(24, 40, 1000.0), (40, 64, 700.0), (30, 90, 500.0)])])
def test_calls_on_different_streams_share_the_tables(cuda_device, interp, shapes):
    """Each accumulator computes on a stream of its own and returns from add() before its work is done; a
    table built for the next one must wait for that work.  Against the same points in one call, the sums in another
    order: 1e-12 of the level's largest |f|."""
    chunks = [uniform_ball(30000, 500.0, seed=k) for k in range(3)]
    for (lmax, nmax, rmax), got in zip(shapes, _interleaved(shapes, chunks, interp)):
        one = catana.sfb_decomposition(catana.PointContainer(np.concatenate(chunks)), lmax, nmax, rmax, True, False,
                                       interpolation=interp)
        for l in range(lmax):
            assert np.max(np.abs(got.f_lmn[l] - one.f_lmn[l])) <= 1e-12 * np.max(np.abs(one.f_lmn[l])), (nmax, l)


def test_raw_calls_on_two_streams(cuda_device):
    """catana_gpu_sfb_raw_dev without weights returns at once: two streams with unlike nmax, in turn, without a
    place for f_lmn of their own."""
    torch = pytest.importorskip("torch")
    pts = torch.from_numpy(uniform_ball(60000, 1000.0, seed=1)).cuda()
    shapes = [(32, 64), (32, 20)]
    streams = [torch.cuda.Stream() for _ in shapes]

    def call(lmax, nmax, st):
        k, c = (torch.zeros(lmax * nmax, dtype=torch.float64, device="cuda") for _ in range(2))
        torch.cuda.current_stream().synchronize()  # zeroed on the default stream
        p = [t.data_ptr() for t in (pts, k, c)]
        _lib.check(_lib.lib.catana_gpu_sfb_raw_dev(p[0], None, 60000, lmax, nmax, 1000.0, _lib.JL_INTERP, p[1], p[2], None, None,
                                                   st.cuda_stream))
        return k, c  # both are held until the work is done

    ref = []
    for s, st in zip(shapes, streams):
        ref.append(call(*s, st))
        torch.cuda.synchronize()
    for _ in range(3):
        got = [call(*s, st) for s, st in zip(shapes, streams)]
        torch.cuda.synchronize()
        assert all(torch.equal(a[1], b[1]) for a, b in zip(got, ref))


@pytest.mark.parametrize("nside,n", [(1, 31), (2, 257), (16, 1000), (64, 20000), (128, 3000)])
def test_every_entry_of_a_pixelized_catalog_is_counted(cuda_device, nside, n):
    """l = 0 holds every point with the same angular factor: its sums over pixels are those over the points, however
    the lanes of a warp part in the bisection for their pixels (clumped and empty pixels, partial warps).  Only
    the order of the sums differs: 1e-12."""
    pts = uniform_ball(n, 1000.0, seed=nside)
    pts[: n // 3, 1:] = [0.3, 1.0]  # a third of the points in one pixel
    raw = catana.sfb_decomposition(catana.PointContainer(pts), 1, 8, 1000.0, True, False, interpolation="off")
    ppc = catana.PixelizedPointContainer(nside, catana.PointContainer(pts))
    hpx = catana.sfb_decomposition(ppc, 1, 8, 1000.0, True, False, interpolation="off")
    assert np.max(np.abs(hpx.f_lmn[0] - raw.f_lmn[0])) <= 1e-12 * np.max(np.abs(raw.f_lmn[0]))


@pytest.mark.parametrize("n,power", [(300, -966), (300, -980), (40, -1000), (3, 1020), (2, 1022)])
def test_weights_at_the_ends_of_the_double_range(cuda_device, n, power):
    """f is normalised by the weights' sum, so weights times a power of two change it by the rounding of numbers near
    the end of FP64's range only: sums of ~2^-1000 times products of ~2^-20 keep 2^-1074 + 1020 of their own, 1e-12
    of the level's largest |f|."""
    pts = uniform_ball(n, 1.0, seed=n)
    w = np.random.default_rng(n).uniform(0.5, 1.0, n)
    args = (11, 4, 1.0, True, False)
    a = catana.sfb_decomposition(catana.PointContainer(pts), *args, weights=w, interpolation="on")
    b = catana.sfb_decomposition(catana.PointContainer(pts), *args, weights=np.ldexp(w, power), interpolation="on")
    for l, (f, g) in enumerate(zip(a.f_lmn, b.f_lmn)):
        assert np.max(np.abs(f - g)) <= 1e-12 * np.max(np.abs(f)), l


def _entries(pts, w, lmax, nmax):
    """f_lmn of the weighted catalog by every entry that takes weights."""
    torch = pytest.importorskip("torch")
    pc = catana.PointContainer(pts)
    yield catana.sfb_decomposition(pc, lmax, nmax, 1.0, True, False, weights=w, interpolation="on").f_lmn
    yield catana.sfb_decomposition_batched([pc, pc], lmax, nmax, 1.0, weights=[None, w], store_flmn=True, verbose=False,
                                           precision="plain", interpolation="on")[1].f_lmn
    with catana.SFBAccumulator(lmax, nmax, 1.0, precision="plain", interpolation="on") as acc:
        acc.add(pts, w)
        yield acc.finish(store_flmn=True).f_lmn
    d = [torch.from_numpy(a).cuda() for a in (pts, w)]
    k, c = (torch.zeros(lmax * nmax, dtype=torch.float64, device="cuda") for _ in range(2))
    f = torch.zeros(nmax * lmax * (lmax + 1) // 2, dtype=torch.complex128, device="cuda")
    _lib.check(_lib.lib.catana_gpu_sfb_raw_dev(d[0].data_ptr(), d[1].data_ptr(), len(pts), lmax, nmax, 1.0, _lib.JL_INTERP,
                                               k.data_ptr(), c.data_ptr(), f.data_ptr(), None, None))
    f = f.cpu().numpy()
    yield [f[nmax * l * (l + 1) // 2: nmax * (l + 1) * (l + 2) // 2].reshape(l + 1, nmax) for l in range(lmax)]


@pytest.mark.parametrize("power", [0, 7, 8, 9, 20, 45, 70])
def test_light_points_beside_a_heavy_one(cuda_device, power):
    """A heavy point at a pole adds nothing to m > 0: those modes are the light points' alone, and as accurate as
    without it.  Fixed-point terms are cut at 2^-55 of the heaviest weight's bound, so up to the 2^8 that they are taken for
    a mode errs by sqrt(33) 2^(8 - 55), times what the bound exceeds a mode's largest term by (below 2^5 here): 2e-12
    of the mode's largest order."""
    lmax, nmax = 8, 4
    pts = uniform_ball(33, 1.0, seed=4)
    pts[5, 1] = 0.0
    w = np.random.default_rng(2).uniform(0.75, 1.0, 33)
    light = w.copy()
    light[5] = 0.0
    w[5] = 0.75 * 2.0 ** power
    ref = catana.sfb_decomposition(catana.PointContainer(pts), lmax, nmax, 1.0, True, False, weights=light, interpolation="on")
    for f in _entries(pts, w, lmax, nmax):
        for l in range(1, lmax):
            g = ref.f_lmn[l] * (light.sum() / w.sum())
            for m in range(1, l + 1):
                assert np.max(np.abs(f[l][m] - g[m])) <= 2e-12 * np.max(np.abs(g[m])), (l, m)


class _AllocLimit:
    """Within it, no internal buffer of more than `bytes` can be had."""

    def __init__(self, nbytes):
        self.nbytes = nbytes

    def __enter__(self):
        _lib.lib.catana_gpu_test_alloc_limit(self.nbytes)

    def __exit__(self, *exc):
        _lib.lib.catana_gpu_test_alloc_limit(0)


@pytest.mark.parametrize("interp,precision,lmax,nmax,limit", [("on", "plain", 90, 30, 4 << 20), ("poly", "plain", 200, 4, 4 << 20),
                                                              ("auto", "split", 200, 4, 2 << 20)])
def test_a_table_that_could_not_be_had_is_not_taken_for_cached(cuda_device, interp, precision, lmax, nmax, limit):
    """A failed growth frees the buffer that a table was cached in: the next call of the old size builds it again.
    The limits lie between the catalog's and the results' buffers (at most 2.0, 1.3, 1.3 MB) and the tables (21.6, 4.4,
    2.1 MB).  Tables for other l ranges are rounded otherwise (j_l of all l by one recurrence): to ~1e-14 the
    polynomials in FP64, to ~1e-7 those of the split form."""
    pts = uniform_ball(2000, 1000.0, seed=3)

    def call(lmax, nmax):
        return catana.sfb_decomposition(catana.PointContainer(pts), lmax, nmax, 1000.0, True, False, interpolation=interp,
                                        precision=precision)

    call(lmax, nmax)  # what this and the next call share is there
    before = call(6, 5)
    with _AllocLimit(limit):
        with pytest.raises(MemoryError):
            call(lmax + 20, nmax + 1)
    after = call(6, 5)
    assert np.allclose(before.c_ln, after.c_ln, rtol=1e-5 if precision == "split" else 1e-12, atol=0.0)


def test_a_pixelized_workspace_goes_by_the_entries(cuda_device):
    """200k points in the 12 pixels of nside 1 are 3.1k entries: the sort takes 6.5 MB, rows and phases 3 MB (by the points
    they took 154), so 16 MB are enough, to the same bits."""
    pts = uniform_ball(200000, 1000.0, seed=1)
    ppc = catana.PixelizedPointContainer(1, catana.PointContainer(pts))

    def call():
        return catana.sfb_decomposition(ppc, 24, 4, 1000.0, True, False)

    ref = call()
    with _AllocLimit(16 << 20):
        got = call()
    assert np.array_equal(got.c_ln, ref.c_ln)


def test_one_level_of_many_radial_orders_is_cut_too(cuda_device):
    """300k points with 1000 radial orders have 2.4 GB of j_l in one level; a pass takes as many points as keep it under
    2 GB.  The catalog's sums are those of its halves, in another order: 1e-12 of the level's largest |f|."""
    n, lmax, nmax = 300000, 2, 1000
    pts = uniform_ball(n, 1000.0, seed=2)

    def call(p):
        return catana.sfb_decomposition(catana.PointContainer(p), lmax, nmax, 1000.0, True, False, interpolation="poly").f_lmn

    with _AllocLimit(2100 << 20):
        whole = call(pts)
    halves = [call(pts[: n // 2]), call(pts[n // 2:])]
    for l in range(lmax):
        both = 0.5 * (halves[0][l] + halves[1][l])
        assert np.max(np.abs(whole[l] - both)) <= 1e-12 * np.max(np.abs(both)), l


def _launches(call):
    n = _lib.lib.catana_gpu_launch_count()
    return call(), _lib.lib.catana_gpu_launch_count() - n


@pytest.mark.parametrize("n,lmax,nmax,limit,interp", [
    # 17 MB of rows and phases: passes of 5208 points
    (20000, 24, 4, 5 << 20, "on"), (20000, 24, 4, 5 << 20, "off"), (20000, 24, 4, 5 << 20, "poly"),
    # tables of 3.8 MB fit, their pair form of 7.7 does not: the FP64 path
    (600, 24, 20, 6 << 20, "on")])
def test_memory_that_cannot_be_had(cuda_device, n, lmax, nmax, limit, interp):
    """Smaller passes, and past them the FP64 path, whose buffers are smaller: the sums in another order, and with the
    FP64 path another table position (4e-14 of j_l's envelope) and recurrence: 1e-12 of the level's largest |f|."""
    pts = uniform_ball(n, 1000.0, seed=n)
    w = np.random.default_rng(n).uniform(0.5, 1.5, n)

    def call(nmax=nmax):
        return catana.sfb_decomposition(catana.PointContainer(pts), lmax, nmax, 1000.0, True, False, weights=w,
                                        interpolation=interp).f_lmn

    call(nmax - 1)  # tables of another nmax: both calls build their own
    ref, few = _launches(call)
    call(nmax - 1)
    with _AllocLimit(limit):
        got, more = _launches(call)
    assert more > few  # more passes, or a launch per level
    for l in range(lmax):
        assert np.max(np.abs(got[l] - ref[l])) <= 1e-12 * np.max(np.abs(ref[l])), l


@pytest.mark.parametrize("nside,n,lmax,nmax,limit", [(32, 40000, 24, 4, 5 << 20), (4, 3000, 10, 6, 800 << 10)])
def test_memory_that_cannot_be_had_pixelized(cuda_device, nside, n, lmax, nmax, limit):
    """The same for the pixelized sum: 12k entries in passes; room for the tables
    (0.5 MB) but not for their pair form, so the maps."""
    ppc = catana.PixelizedPointContainer(nside, catana.PointContainer(uniform_ball(n, 1000.0, seed=n)))

    def call(nmax=nmax):
        return catana.sfb_decomposition(ppc, lmax, nmax, 1000.0, True, False).f_lmn

    call(nmax - 1)
    ref, few = _launches(call)
    call(nmax - 1)
    with _AllocLimit(limit):
        got, more = _launches(call)
    assert more > few  # more passes, or a launch per level
    fmax = max(np.max(np.abs(f)) for f in ref)
    for l in range(lmax):
        assert np.max(np.abs(got[l] - ref[l])) <= 1e-12 * fmax, l


@pytest.mark.parametrize("n,lmax,nmax,fp64", [(100, 80, 600, True), (2, 300, 200, True), (20, 1, 16, True), (300, 100, 64, False),
                                              (100, 512, 64, False), (4000, 70, 300, False), (300, 6, 64, False)])
def test_the_faster_path_for_few_points(cuda_device, n, lmax, nmax, fp64):
    """The FP64 path launches two kernels a level, the tensor-core path at most three dozen for these in all; levels
    below 4 agree with the other side's oracle in either."""
    from oracle import oracle as O
    pts = uniform_ball(n, 1000.0, seed=n)

    def call():
        return catana.sfb_decomposition(catana.PointContainer(pts), lmax, nmax, 1000.0, True, False, interpolation="on")

    call()
    res, launches = _launches(call)
    assert (launches >= 2 * lmax + 1 and launches < 2 * lmax + 5) == fp64, launches
    keep = min(lmax, 4)
    f = O.sfb_raw(pts, keep, nmax, 1000.0, interpolated=True)[2]
    for l in range(keep):
        assert np.max(np.abs(res.f_lmn[l] - f[l])) <= 1e-10 * np.max(np.abs(f[l])), l


@pytest.mark.parametrize("nside,n,lmax,nmax,maps", [(1, 3, 24, 1500, True), (4, 300, 24, 1500, True), (1, 300, 24, 8, False),
                                                    (32, 2000, 24, 8, False), (16, 20000, 12, 300, False)])
@pytest.mark.parametrize("interp", ["on", "off"])
def test_the_faster_path_for_few_pixelized_points(cuda_device, nside, n, lmax, nmax, maps, interp):
    """The maps launch at least four kernels a level, the sum over entries at most three dozen for these in all; the lowest
    levels agree with the oracle in either."""
    from oracle import oracle as O
    if interp == "off" and (maps and n > 3 or nmax == 300):
        return  # exact j_l: another crossing point
    ppc = catana.PixelizedPointContainer(nside, catana.PointContainer(uniform_ball(n, 1000.0, seed=n)))

    def call():
        return catana.sfb_decomposition(ppc, lmax, nmax, 1000.0, True, False, interpolation=interp)

    call()
    res, launches = _launches(call)
    assert (launches >= 4 * lmax) == maps, launches
    f = O.sfb_healpix(nside, ppc.offsets, ppc.r_sorted, 2, nmax, 1000.0, interpolated=interp == "on")[2]
    for l in range(2):
        assert np.max(np.abs(res.f_lmn[l] - f[l])) <= 1e-10 * np.max(np.abs(f[l])), l


@pytest.mark.parametrize("lmax,nmax", [(1, 1), (3, 200), (520, 2)])
def test_an_empty_pixelized_catalog(cuda_device, lmax, nmax):
    """No point on any path: the normalisation's 1 / N times 0, as in the reference."""
    ppc = catana.PixelizedPointContainer(4)
    ppc.offsets, ppc.r_sorted = np.zeros(12 * 16 + 1, dtype=np.int64), np.zeros(0)
    res = catana.sfb_decomposition(ppc, lmax, nmax, 1000.0, True, False)
    assert np.all(np.isnan(res.c_ln)) and all(np.all(np.isnan(f)) for f in res.f_lmn)
