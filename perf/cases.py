"""Workloads of the framework's public entry points, with inputs, work counts and values in 64 bits.

What a user of this package runs: the plain (drop-in) SFB decomposition of a catalog, from a
few hundred points to survey subsamples and mock catalogs; its HEALPix form, which also bins the
catalog; the tensor-core forms on a large catalog, on a batch of catalogs and on a catalog
streamed in float32 chunks; and, around them, the record ingest and the shot-noise integrals.
Sizes follow the workloads of this repository's benchmark and tests; the largest are cut so that
a pass stays below a second.

A case is a dict of plain values; `family` names the entry point.  Catalogs are points uniform
in a ball, the survey's are n(r) ~ r^2 exp(-(r/300)^2) with a galactic cut, the HEALPix ones
carry 10% of their points in clumps -- each as in the benchmark.

The split forms hold every operand and running sum in FP32 or less and return FP64 containers;
which FP32 sums they form depends on a schedule that is timed at run time (batched) or cut to the
chip (the others), so two processes agree to FP32 rounding only.  Their C_ln and f_lmn are handed
on in float32, the precision that they carry; k_ln stays float64.
"""
import ctypes
import math

import numpy as np
import torch

import catana_gb300 as catana
from catana_gb300 import _lib
from catana_gb300 import besseltools

RMAX = 1000.0

_SPLIT = ("split", "split_accurate")
_FORM = {"plain": _lib.FORM_PLAIN, "split": _lib.FORM_SPLIT,
         "split_accurate": _lib.FORM_SPLIT | _lib.SPLIT_ACCURATE}
_JL = {"auto": _lib.JL_AUTO, "on": _lib.JL_INTERP, "off": _lib.JL_EXACT, "poly": _lib.JL_POLY}


def _raw(n, lmax, nmax, interp="auto", weights=False, **kw):
    return dict(family="raw", n=n, lmax=lmax, nmax=nmax, interp=interp, weights=weights, **kw)


def _dev(n, lmax, nmax, precision="plain", interp="auto", weights=True, **kw):
    return dict(family="raw_dev", n=n, lmax=lmax, nmax=nmax, precision=precision, interp=interp, weights=weights, **kw)


def listed():
    return [
        # the reference's own test catalog in size: a few hundred points, exact j_l (the rule for
        # N <= 1000); a notebook or test-suite call, where launches and host time count
        _raw(445, 10, 10, name="raw_445_l10_n10"),
        # a galaxy-group or cluster subsample through the default call (interpolated j_l)
        _raw(5000, 24, 20, name="raw_5k_l24_n20"),
        # the plain decomposition of one mock catalog: the benchmark's FP64 workload
        _raw(100000, 32, 32, name="raw_100k_l32_n32"),
        # a weighted survey subsample at higher resolution, arrays already on the device
        _dev(200003, 96, 48, name="dev_200k_l96_n48_w"),
        # the FP64 yardstick of the split forms: j_l without table error
        _dev(60000, 128, 64, interp="poly", name="dev_poly_60k_l128_n64_w"),
        # the pixelized decomposition: the benchmark's HEALPix workload
        dict(family="healpix", nside=256, n=1000000, lmax=128, nmax=64, reverse=False, name="healpix_256_1M_l128_n64"),
        # binning that workload's catalog, as every HEALPix user does once per catalog
        dict(family="bin", nside=256, n=1000000, name="bin_256_1M"),
        # a tenth of the headline split-precision workload at its lmax, nmax and weights
        _dev(1000000, 256, 128, precision="split", name="split_1M_l256_n128_w"),
        # mock catalogs of uneven size, lmax and rmax in one call with a kmax cut
        dict(family="batched", ncat=8, nmin=10000, nmaxp=200000, kmax=0.2, nmax=128, precision="split", name="batched_8_k0.2"),
        # the masked survey streamed in float32 chunks at lmax 512, nmax 256
        dict(family="stream", chunks=2, chunk=20000, lmax=512, nmax=256, precision="split", name="stream_2x20k_l512_n256"),
        # reading a survey: float32 Cartesian records through window and mask
        dict(family="ingest", n=4000000, f32=True, cartesian=True, nside=64, name="ingest_4M_f32"),
        # one multipole of the shot-noise matrix: all (n1, n2) pairs of a window table
        dict(family="integrals", l=16, nk=32, nodes=10001, rmax=1000.0, name="shotnoise_l16_32x32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    f = rng.choice(["raw", "raw", "raw_dev", "poly", "exact", "healpix", "bin", "split", "split", "batched", "stream",
                    "ingest", "integrals"])
    if f == "raw":
        lmax, nmax = _log(rng, 6, 64), _log(rng, 5, 64)
        n = min(_log(rng, 300, 150000), int(4e10 / (nmax * lmax * (lmax + 1) / 2)))
        return _raw(n, lmax, nmax, "auto", rng.random() < 0.3)
    if f == "raw_dev":
        lmax, nmax = _log(rng, 24, 160), _log(rng, 16, 130)
        n = min(_log(rng, 5000, 250000), int(4e10 / (nmax * lmax * (lmax + 1) / 2)))
        return _dev(n, lmax, nmax, "plain", "on", rng.random() < 0.7)
    if f == "poly":
        lmax, nmax = _log(rng, 24, 160), _log(rng, 16, 130)
        n = min(_log(rng, 3000, 100000), int(4e10 / (nmax * lmax * (lmax + 1) / 2)))
        return _dev(n, lmax, nmax, "plain", "poly", rng.random() < 0.5)
    if f == "exact":
        lmax, nmax = _log(rng, 6, 48), _log(rng, 5, 40)
        n = min(_log(rng, 300, 20000), int(2e9 / (nmax * lmax * (lmax + 1) / 2)))
        return _raw(n, lmax, nmax, "off", rng.random() < 0.3)
    if f == "healpix":
        nside = rng.choice([32, 64, 128, 256])
        lmax = min(_log(rng, 10, 128), 2 * nside)
        return dict(family="healpix", nside=nside, n=_log(rng, 2000, 1000000), lmax=lmax, nmax=_log(rng, 8, 64),
                    reverse=rng.random() < 0.3)
    if f == "bin":
        return dict(family="bin", nside=rng.choice([16, 64, 256, 512]), n=_log(rng, 1000, 4000000))
    if f == "split":
        lmax, nmax = _log(rng, 48, 256), _log(rng, 24, 128)
        n = min(_log(rng, 10000, 1000000), int(4e12 / (nmax * lmax * (lmax + 1) / 2)))
        return _dev(n, lmax, nmax, rng.choice(["split", "split", "split_accurate"]), "auto", rng.random() < 0.7)
    if f == "batched":
        return dict(family="batched", ncat=rng.randint(2, 16), nmin=_log(rng, 2000, 20000),
                    nmaxp=_log(rng, 30000, 200000), kmax=rng.choice([0.0, 0.1, 0.2]), nmax=_log(rng, 32, 128),
                    precision="split")
    if f == "stream":
        return dict(family="stream", chunks=rng.randint(1, 3), chunk=_log(rng, 4000, 20000), lmax=_log(rng, 128, 512),
                    nmax=_log(rng, 64, 256), precision="split")
    if f == "ingest":
        return dict(family="ingest", n=_log(rng, 10000, 4000000), f32=rng.random() < 0.7, cartesian=rng.random() < 0.6,
                    nside=rng.choice([0, 16, 64]))
    return dict(family="integrals", l=_log(rng, 1, 128) - 1, nk=_log(rng, 4, 36), nodes=_log(rng, 1001, 20001),
                rmax=float(_log(rng, 100, 1500)))


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
def _gen(seed, stream=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + stream)
    return g


def _uni(g, n, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(n, generator=g, device="cuda", dtype=torch.float64)


def _ball(g, n, rmax):
    """(r, theta, phi) uniform in a ball."""
    r = rmax * _uni(g, n) ** (1.0 / 3.0)
    th = torch.acos(_uni(g, n, -1.0, 1.0))
    return torch.stack([r, th, _uni(g, n, 0.0, 2.0 * math.pi)], 1).contiguous()


def _spherical(xyz):
    x, y, z = xyz[:, 0], xyz[:, 1], xyz[:, 2]
    rho = torch.sqrt(x * x + y * y)
    ph = torch.atan2(y, x)
    return torch.stack([torch.sqrt(rho * rho + z * z), torch.atan2(rho, z), torch.where(ph < 0, ph + 2 * math.pi, ph)],
                       1).contiguous()


def _clumpy(g, n, rmax):
    """90% uniform in the ball, 10% in 1000 Gaussian clumps of sigma 5."""
    nc = n // 10
    p = _ball(g, n - nc, rmax)
    c = _ball(g, 1000, 0.97 * rmax)
    st = torch.sin(c[:, 1])
    cx = torch.stack([c[:, 0] * st * torch.cos(c[:, 2]), c[:, 0] * st * torch.sin(c[:, 2]), c[:, 0] * torch.cos(c[:, 1])], 1)
    at = (_uni(g, nc) * 1000).long().clamp_(max=999)
    q = _spherical(cx[at] + 5.0 * torch.randn(nc, 3, generator=g, device="cuda", dtype=torch.float64))
    q[:, 0].clamp_(max=0.9999 * rmax)
    return torch.cat([p, q]).contiguous()


def _survey(g, n, rmax=1500.0, a=300.0):
    """Radial selection r^2 exp(-(r/a)^2) below rmax, |theta - pi/2| > 20 degrees; float32."""
    z = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64) * (a / math.sqrt(2.0))
    r = z.square().sum(1).sqrt().clamp_(max=0.999 * rmax)
    u = _uni(g, n, math.sin(math.radians(20.0)), 1.0)
    s = torch.where(_uni(g, n) < 0.5, -1.0, 1.0)
    return torch.stack([r, torch.acos(s * u), _uni(g, n, 0.0, 2.0 * math.pi)], 1).float().contiguous()


def _records(g, case):
    """Survey records: of ten, two lie beyond the radial cut and two in the masked band |z| < 0.34 r, so
    the number of survivors does not depend on the seed."""
    n = case["n"]
    i = torch.arange(n, device="cuda") % 10
    r = torch.where((i == 6) | (i == 7), _uni(g, n, 1600.0, 2500.0), 1450.0 * _uni(g, n) ** (1.0 / 3.0))
    ct = torch.where(i >= 8, _uni(g, n, -0.25, 0.25), _uni(g, n, 0.45, 1.0) * torch.where(_uni(g, n) < 0.5, -1.0, 1.0))
    ph = _uni(g, n, 0.0, 2.0 * math.pi)
    if not case["cartesian"]:
        return torch.stack([r, torch.acos(ct), ph], 1)
    st = torch.sqrt(1.0 - ct * ct)
    return torch.stack([r * st * torch.cos(ph), r * st * torch.sin(ph), r * ct], 1)


def _band_mask(nside):
    """1 outside the band |cos(theta)| < 0.34, per RING pixel."""
    npx, x, _, _ = _ring_geometry(nside)
    return torch.repeat_interleave((x.abs() >= 0.34).float(), npx)


def _catalogs(case):
    """Sizes, lmax and rmax of the batch: log-uniform sizes, lmax 64..200, rmax 500..1500."""
    out = []
    for i in range(case["ncat"]):
        t = (i + 0.5) / case["ncat"]
        n = int(round(math.exp(math.log(case["nmin"]) + t * (math.log(case["nmaxp"]) - math.log(case["nmin"])))))
        out.append((n, 64 + (i * 53) % 137, 500.0 + (i * 379.0) % 1000.0))
    return out


def _pd(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def prepare(case, seed):
    f, g = case["family"], _gen(seed)
    s = {"case": case}
    if f == "raw":
        s["pc"] = catana.PointContainer(_ball(g, case["n"], RMAX).cpu().numpy())
        s["w"] = _uni(g, case["n"], 0.5, 1.5).cpu().numpy() if case["weights"] else None
    elif f == "raw_dev":
        lm, fs = case["lmax"] * case["nmax"], case["nmax"] * case["lmax"] * (case["lmax"] + 1) // 2
        s["pts"] = _ball(g, case["n"], RMAX)
        s["w"] = _uni(g, case["n"], 0.5, 1.5) if case["weights"] else None
        s["k"], s["c"] = (torch.zeros(lm, dtype=torch.float64, device="cuda") for _ in range(2))
        s["f"] = torch.zeros(2 * fs, dtype=torch.float64, device="cuda")
        s["flags"] = _FORM[case["precision"]] | _JL[case["interp"]]
    elif f == "healpix":
        pts = _clumpy(g, case["n"], RMAX).cpu().numpy()
        s["ppc"] = catana.PixelizedPointContainer(case["nside"], catana.PointContainer(pts))
        lm, fs = (case["lmax"], case["nmax"]), case["nmax"] * case["lmax"] * (case["lmax"] + 1) // 2
        s["k"], s["c"], s["f"] = np.zeros(lm), np.zeros(lm), np.zeros(fs, dtype=np.complex128)
    elif f == "bin":
        s["pc"] = catana.PointContainer(_clumpy(g, case["n"], RMAX).cpu().numpy())
    elif f == "batched":
        s["cats"] = [catana.PointContainer(_ball(_gen(seed, i + 1), n, r).cpu().numpy())
                     for i, (n, _, r) in enumerate(_catalogs(case))]
        s["lmax"], s["rmax"] = [c[1] for c in _catalogs(case)], [c[2] for c in _catalogs(case)]
    elif f == "stream":
        s["chunks"] = [_survey(_gen(seed, i + 1), case["chunk"] + 7 * i).cpu().pin_memory().numpy()
                       for i in range(case["chunks"])]
    elif f == "ingest":
        rec = _records(g, case)
        s["rec"] = (rec.float() if case["f32"] else rec).cpu().numpy()
        s["kw"] = dict(coordinate_type="cartesian" if case["cartesian"] else "spherical", tophat_r0=1500.0)
        if case["nside"]:
            s["kw"]["mask"] = _band_mask(case["nside"]).cpu().numpy()
    elif f == "integrals":
        # the window differs with the seed, the wave numbers are k_ln of this l
        a = 0.3 + 0.2 * float(_uni(g, 1).cpu())
        r = case["rmax"]
        s["w"] = catana.FunctionInterpolator(lambda x: np.exp(-(x / (a * r)) ** 2) * x ** 2, case["nodes"], 0.0, r)
        k = catana.compute_kln(case["l"] + 1, case["nk"], r)[case["l"]]
        s["k1"], s["k2"] = np.meshgrid(k, k)
    return s


def run(s):
    case = s["case"]
    f = case["family"]
    if f == "raw":
        r = catana.sfb_decomposition(s["pc"], case["lmax"], case["nmax"], RMAX, True, False, weights=s["w"],
                                     interpolation=case["interp"])
        # one packed array where the list of multipoles is long
        fl = list(r.f_lmn) if case["lmax"] <= 32 else np.concatenate([x.reshape(-1) for x in r.f_lmn])
        return {"k_ln": r.k_ln, "c_ln": r.c_ln, "f_lmn": fl}
    if f == "raw_dev":
        st = _lib.lib.catana_gpu_sfb_raw_dev(_pd(s["pts"]), _pd(s["w"]), case["n"], case["lmax"], case["nmax"], RMAX,
                                             s["flags"], _pd(s["k"]), _pd(s["c"]), _pd(s["f"]), None,
                                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        _lib.check(st, "sfb_raw_dev")
        if case["precision"] in _SPLIT:
            return {"k_ln": s["k"], "c_ln": s["c"].float(), "f_lmn": s["f"].float()}
        return {"k_ln": s["k"], "c_ln": s["c"], "f_lmn": s["f"]}
    if f == "healpix":
        p = s["ppc"]
        fn = _lib.lib.catana_gpu_sfb_reverse if case["reverse"] else _lib.lib.catana_gpu_sfb_healpix
        _lib.check(fn(p.nside, _lib.ptr(p.offsets), _lib.ptr(p.r_sorted), case["lmax"], case["nmax"], RMAX,
                      _lib.JL_INTERP, _lib.ptr(s["k"]), _lib.ptr(s["c"]), _lib.ptr(s["f"]), None), "sfb_healpix")
        return {"k_ln": s["k"], "c_ln": s["c"], "f_lmn": s["f"]}
    if f == "bin":
        p = catana.PixelizedPointContainer(case["nside"], s["pc"])
        return {"offsets": p.offsets, "r": p.r_sorted}
    if f == "batched":
        r = catana.sfb_decomposition_batched(s["cats"], s["lmax"], case["nmax"], s["rmax"], kmax=case["kmax"],
                                             verbose=False, precision=case["precision"])
        return [{"k_ln": x.k_ln, "c_ln": x.c_ln.astype(np.float32)} for x in r]
    if f == "stream":
        with catana.SFBAccumulator(case["lmax"], case["nmax"], 1500.0, precision=case["precision"]) as acc:
            for c in s["chunks"]:
                acc.add(c)
            r = acc.finish()
        return {"k_ln": r.k_ln, "c_ln": r.c_ln.astype(np.float32)}
    if f == "ingest":
        return np.asarray(catana.ingest(s["rec"], **s["kw"]))
    return besseltools.double_sbessel_integrator(s["w"], case["l"], case["rmax"], s["k1"], s["k2"])


def _modes(lmax, nmax):
    return nmax * lmax * (lmax + 1) // 2


def work(case):
    f = case["family"]
    if f in ("raw", "raw_dev"):
        m = _modes(case["lmax"], case["nmax"])
        b = case["n"] * (32 if case["weights"] else 24) + 16 * m + 16 * case["lmax"] * case["nmax"]
        return {"bytes": b, "flops": 4.0 * case["n"] * m}
    if f == "healpix":
        # a ring transform of each pixel map (5 N log2 N on pairs of real rows), the maps and the ring sums
        npix, L, M = 12 * case["nside"] ** 2, case["lmax"], case["nmax"]
        fl = L * M * (4.0 * case["n"] + 2.5 * npix * math.log2(4 * case["nside"])) + 8.0 * 4 * case["nside"] * _modes(L, M)
        return {"bytes": 8 * case["n"] + 8 * npix + 16 * _modes(L, M) + 16 * L * M, "flops": fl}
    if f == "bin":
        return {"bytes": case["n"] * 32 + 8 * 12 * case["nside"] ** 2, "flops": 0}
    if f == "batched":
        b = fl = 0
        for n, lmax, rmax in _catalogs(case):
            # n-th zero of j_l ~ l + 1.86 l^(1/3) + pi n: the radial orders that the cut keeps
            for l in range(lmax):
                top = case["kmax"] * rmax if case["kmax"] else 1e9
                live = max(0, min(case["nmax"], int((top - l - 1.86 * l ** (1 / 3.0)) / math.pi)))
                fl += 4.0 * n * live * (l + 1)
            b += 24 * n + 16 * lmax * case["nmax"]
        return {"bytes": b, "flops": fl}
    if f == "stream":
        n = case["chunks"] * case["chunk"]
        return {"bytes": 12 * n + 16 * case["lmax"] * case["nmax"], "flops": 4.0 * n * _modes(case["lmax"], case["nmax"])}
    if f == "ingest":
        return {"bytes": case["n"] * ((12 if case["f32"] else 24) + 9) + 48 * case["nside"] ** 2, "flops": 0}
    # each table segment of each pair at least once: w, both j_l and the sum
    return {"bytes": 8 * case["nodes"] + 24 * case["nk"] ** 2, "flops": 4.0 * case["nk"] ** 2 * case["nodes"]}


# ---------------------------------------------------------------------------------------
# the same values in 64 bits, from plain torch and numpy
# ---------------------------------------------------------------------------------------
def _jl_pair(l, z):
    """j_l(z), j_{l+1}(z) for vectors l (ascending, 0, 1, 2, ...) and z > l, by upward recurrence."""
    j0 = np.sin(z) / z
    j1 = (j0 - np.cos(z)) / z
    a, b = j0.copy(), j1.copy()
    p, c = j0, j1
    for k in range(1, l.size):
        n = (2.0 * k + 1.0) / z[k:] * c[-(l.size - k):] - p[-(l.size - k):]
        p = c[-(l.size - k):]
        c = n
        a[k], b[k] = p[0], c[0]
    return a, b


def _zeros(lmax, count):
    """Zeros 0..count-1 of j_l, l < lmax: the reference's guesses, Newton step and stopping rule."""
    l = np.arange(lmax, dtype=np.float64)
    h = l + 0.5
    g = [h + 1.8557571 * h ** (1 / 3.) + 1.033150 * h ** (-1 / 3.) - 0.00397 / h - 0.0908 * h ** (-5 / 3.) + 0.043 * h ** (-7 / 3.),
         h + 3.2446076 * h ** (1 / 3.) + 3.158244 * h ** (-1 / 3.) - 0.08331 / h - 0.8437 * h ** (-5 / 3.) + 0.864 * h ** (-7 / 3.)]
    g[0][0], g[1][0] = math.pi, 2.0 * math.pi
    out = np.zeros((lmax, count))

    def newton(z):
        live = np.ones(lmax, dtype=bool)
        while live.any():
            j, j1 = _jl_pair(l, z)
            d = j / (l / z * j - j1)
            z = np.where(live, z - d, z)
            live &= d / z > 1e-15
        return z

    for n in range(count):
        out[:, n] = newton(g[n].copy() if n < 2 else 2 * out[:, n - 1] - out[:, n - 2])
    return out


def _jl_table(lmax, x, only=None):
    """j_l(x) for l < lmax as [lmax, len(x)] (or the row of l = only), x >= 0 on the device: upward for
    l <= x, downward ratios j_k / j_{k-1} beyond."""
    top = (lmax if only is None else only + 1)
    xs = torch.where(x > 0, x, torch.full_like(x, 1e-300))
    r = torch.zeros_like(xs)
    ratio = torch.zeros(top + 1, xs.numel(), dtype=torch.float64, device=xs.device)
    for k in range(int(top + 40 + 20 * (top + 1) ** (1 / 3.)), 0, -1):
        r = 1.0 / ((2.0 * k + 1.0) / xs - r)
        if k <= top:
            ratio[k] = r
    out = torch.zeros(top, xs.numel(), dtype=torch.float64, device=xs.device)
    j0 = torch.where(x > 0, torch.sin(xs) / xs, torch.ones_like(xs))
    out[0] = j0
    if top > 1:
        out[1] = torch.where(x >= 1.0, (j0 - torch.cos(xs)) / xs, j0 * ratio[1])
    for k in range(1, top - 1):
        out[k + 1] = torch.where(x >= k + 1.0, (2.0 * k + 1.0) / xs * out[k] - out[k - 1], out[k] * ratio[k + 1])
    return out if only is None else out[only]


_NC = 15


def _cheb_tables(lmax, zmax):
    """Chebyshev coefficients of j_l on unit intervals centred on the integers: [lmax, interval, _NC]."""
    nint = int(math.floor(zmax + 0.5)) + 2
    t = torch.cos((2.0 * torch.arange(_NC, dtype=torch.float64, device="cuda") + 1.0) * math.pi / (2.0 * _NC))
    z = (torch.arange(nint, dtype=torch.float64, device="cuda")[:, None] + 0.5 * t[None, :]).reshape(-1)
    v = _jl_table(lmax, z.abs())
    odd = (torch.arange(lmax, device="cuda") % 2 == 1)[:, None] & (z < 0)[None, :]
    v = torch.where(odd, -v, v).reshape(lmax, nint, _NC)
    r = torch.arange(_NC, dtype=torch.float64, device="cuda")
    dct = torch.cos(r[:, None] * torch.acos(t)[None, :]) * (2.0 / _NC)
    dct[0] *= 0.5
    return v @ dct.T


def _cheb_eval(co, z):
    """j_l(z) from the coefficients [interval, _NC] of one l."""
    zr = torch.round(z)
    i = zr.long()
    t2 = 4.0 * (z - zr)
    b1 = torch.zeros_like(z)
    b2 = torch.zeros_like(z)
    for s in range(_NC - 1, 0, -1):
        b1, b2 = co[:, s].contiguous()[i] + t2 * b1 - b2, b1
    return co[:, 0].contiguous()[i] + 0.5 * t2 * b1 - b2


class _Radial(object):
    """Rows j_l(k_ln r): the linear table of the interpolated branch, or j_l itself."""

    def __init__(self, lmax, nmax, rmax, interp, rtop, zeros=None):
        z = zeros if zeros is not None else _zeros(lmax, max(nmax + 1, 2))
        self.k = z[:lmax, :nmax] / rmax
        self.interp, self.nmax = interp, nmax
        if interp:
            self.ztop = z[:lmax, nmax]
        else:
            self.tab = _cheb_tables(lmax, float(self.k.max()) * rtop + 1.0)

    def rows(self, l, live, r):
        kr = torch.from_numpy(self.k[l, :live]).cuda()[:, None] * r[None, :]
        if not self.interp:
            return _cheb_eval(self.tab[l], kr)
        npts = 1000 * self.nmax
        dx = self.ztop[l] / (npts - 1)
        y = _jl_table(l + 1, torch.arange(npts, dtype=torch.float64, device="cuda") * dx, only=l)
        ia = kr * (1.0 / dx)
        i = ia.long().clamp_(max=npts - 2)
        y0 = y[i]
        return y0 + (y[i + 1] - y0) * (ia - i)


def _legendre(x, lmax):
    """Yields the rows P_lm(x), m = 0..l, of l = 0, 1, ... (spherical-harmonic normalisation)."""
    s = torch.sqrt((1.0 - x) * (1.0 + x))
    p1 = torch.full((1, x.numel()), 1.0 / math.sqrt(4.0 * math.pi), dtype=torch.float64, device=x.device)
    p2 = None
    yield p1
    for l in range(1, lmax):
        m = torch.arange(l - 1, dtype=torch.float64, device=x.device)
        new = torch.empty(l + 1, x.numel(), dtype=torch.float64, device=x.device)
        new[l] = -math.sqrt((2.0 * l + 1.0) / (2.0 * l)) * s * p1[l - 1]
        new[l - 1] = math.sqrt(2.0 * l + 1.0) * x * p1[l - 1]
        if l >= 2:
            a = torch.sqrt((4.0 * l * l - 1.0) / (l * l - m * m))[:, None]
            b = torch.sqrt(((l - 1.0) ** 2 - m * m) / (4.0 * (l - 1.0) ** 2 - 1.0))[:, None]
            new[:l - 1] = a * (x[None, :] * p1[:l - 1] - b * p2[:l - 1])
        p2, p1 = p1, new
        yield new


def _direct(r, x, cos_m, sin_m, w, lmax, rad, norm, kmax=0.0):
    """f = norm k sum_i w_i j_l(k r_i) P_lm(x_i) e^{-i m phi_i} (complex, packed by l) and C_ln."""
    nmax = rad.nmax
    f, c = [], np.zeros((lmax, nmax))
    for l, p in enumerate(_legendre(x, lmax)):
        live = nmax if not kmax else int((rad.k[l] <= kmax).sum())
        fl = np.zeros((l + 1, nmax), dtype=np.complex128)
        if live:
            acc = torch.zeros(2, l + 1, live, dtype=torch.float64, device="cuda")
            step = max(1024, int(3e7 / live))
            for i in range(0, r.numel(), step):
                j = rad.rows(l, live, r[i:i + step])
                if w is not None:
                    j = j * w[None, i:i + step]
                acc[0] += (p[:, i:i + step] * cos_m[:l + 1, i:i + step]) @ j.T
                acc[1] -= (p[:, i:i + step] * sin_m[:l + 1, i:i + step]) @ j.T
            acc = (acc * norm * torch.from_numpy(rad.k[l, :live]).cuda()).cpu().numpy()
            fl[:, :live] = acc[0] + 1j * acc[1]
        f.append(fl)
        a2 = fl.real ** 2 + fl.imag ** 2
        c[l] = (2.0 * a2.sum(0) - a2[0]) / (2 * l + 1)
    return f, c


def _phases(phi, lmax):
    m = torch.arange(lmax, dtype=torch.float64, device="cuda")[:, None]
    a = m * phi[None, :]
    return torch.cos(a), torch.sin(a)


def _norm(rmax, total):
    return math.sqrt(2.0 / math.pi) * 4.0 / 3.0 * math.pi * rmax ** 3 / total


def _ring_pixels(nside, theta, phi):
    """Ring number (0-based), index in the ring of the RING pixel of each direction."""
    z = torch.cos(theta)
    za = z.abs()
    tt = torch.remainder(phi * (2.0 / math.pi), 4.0)
    t1, t2 = nside * (0.5 + tt), nside * z * 0.75
    jp, jm = torch.floor(t1 - t2).long(), torch.floor(t1 + t2).long()
    ir = nside + 1 + jp - jm  # 1 .. 2 nside + 1 from z = 2/3
    kshift = 1 - (ir & 1)
    ip = torch.remainder(torch.div(jp + jm - nside + kshift + 1, 2, rounding_mode="floor"), 4 * nside)
    ring_eq = nside + ir - 2
    tp = tt - torch.floor(tt)
    near = theta.minimum(math.pi - theta) < 0.01
    d = torch.where(near & (za >= 0.99), nside * torch.sin(theta) / torch.sqrt((1.0 + za) / 3.0),
                    nside * torch.sqrt(3.0 * (1.0 - za)))
    q = torch.floor(tp * d).long() + torch.floor((1.0 - tp) * d).long() + 1
    ipc = torch.floor(tt * q).long()
    ipc = torch.where(ipc >= 4 * q, ipc - 4 * q, ipc)
    cap = za > 2.0 / 3.0
    ring = torch.where(cap, torch.where(z > 0, q - 1, 4 * nside - 1 - q), ring_eq)
    return ring, torch.where(cap, ipc, ip)


def _ring_geometry(nside):
    """Per ring: pixels, cos(theta), phi of the first pixel, first pixel number."""
    i = torch.arange(1, 4 * nside, dtype=torch.float64, device="cuda")
    q = torch.minimum(i, 4 * nside - i)
    cap = (i < nside) | (i > 3 * nside)
    npx = torch.where(cap, 4 * q, torch.full_like(q, 4.0 * nside))
    x = torch.where(cap, torch.where(i < nside, 1.0, -1.0) * (1.0 - q * q / (3.0 * nside ** 2)),
                    (2.0 * nside - i) * 2.0 / (3.0 * nside))
    shift = torch.where(cap, torch.full_like(q, 0.5), torch.where((i + nside) % 2 == 0, 0.5, 0.0))
    phi0 = shift * 2.0 * math.pi / npx
    start = torch.cumsum(npx, 0) - npx
    return npx.long(), x, phi0, start.long()


def exact(case, seed):
    f, g = case["family"], _gen(seed)
    if work(case)["flops"] > 6e12:  # minutes in 64 bits
        return None
    if f in ("raw", "raw_dev"):
        L, M = case["lmax"], case["nmax"]
        pts = _ball(g, case["n"], RMAX)
        w = _uni(g, case["n"], 0.5, 1.5) if case["weights"] else None
        interp = case.get("precision", "plain") == "plain" and (
            case["interp"] == "on" or (case["interp"] == "auto" and case["n"] > 1000))
        rad = _Radial(L, M, RMAX, interp, float(pts[:, 0].max()))
        cm, sm = _phases(pts[:, 2], L)
        fl, c = _direct(pts[:, 0].contiguous(), torch.cos(pts[:, 1]), cm, sm, w, L, rad,
                        _norm(RMAX, float(w.sum()) if w is not None else case["n"]))
        if f == "raw" and L <= 32:
            return {"k_ln": rad.k, "c_ln": c, "f_lmn": fl}
        flat = np.concatenate([x.reshape(-1) for x in fl])
        if f == "raw":
            return {"k_ln": rad.k, "c_ln": c, "f_lmn": flat}
        return {"k_ln": rad.k.reshape(-1), "c_ln": c.reshape(-1), "f_lmn": flat.view(np.float64)}
    if f == "healpix":
        L, M, ns = case["lmax"], case["nmax"], case["nside"]
        pts = _clumpy(g, case["n"], RMAX)
        ring, j = _ring_pixels(ns, pts[:, 1], pts[:, 2])
        npx, x, phi0, _ = _ring_geometry(ns)
        N, m = npx[ring][None, :], torch.arange(L, device="cuda")[:, None]
        mm = m % N
        # the frequency read for m: the reference takes F[N - mm] itself past N/2, the dense sum its conjugate
        s = torch.where(2 * mm > N, mm - N if case["reverse"] else N - mm, mm)
        a = m.double() * phi0[ring][None, :] + 2.0 * math.pi * (torch.remainder(j[None, :] * s, N).double() / N.double())
        rad = _Radial(L, M, RMAX, True, RMAX)
        fl, c = _direct(pts[:, 0].contiguous(), x[ring], torch.cos(a), torch.sin(a), None, L, rad, _norm(RMAX, case["n"]))
        return {"k_ln": rad.k, "c_ln": c, "f_lmn": np.concatenate([v.reshape(-1) for v in fl])}
    if f == "bin":
        pts = _clumpy(g, case["n"], RMAX)
        ring, j = _ring_pixels(case["nside"], pts[:, 1], pts[:, 2])
        order = torch.sort(_ring_geometry(case["nside"])[3][ring] + j, stable=True).indices
        return {"offsets": None, "r": pts[order, 0].cpu().numpy()}
    if f == "batched":
        cats = _catalogs(case)
        zeros = _zeros(max(c[1] for c in cats), max(case["nmax"] + 1, 2))
        out = []
        for i, (n, L, rmax) in enumerate(cats):
            pts = _ball(_gen(seed, i + 1), n, rmax)
            rad = _Radial(L, case["nmax"], rmax, False, rmax, zeros)
            cm, sm = _phases(pts[:, 2], L)
            _, c = _direct(pts[:, 0].contiguous(), torch.cos(pts[:, 1]), cm, sm, None, L, rad, _norm(rmax, n), case["kmax"])
            out.append({"k_ln": rad.k, "c_ln": c})
        return out
    if f == "stream":
        L, M = case["lmax"], case["nmax"]
        pts = torch.cat([_survey(_gen(seed, i + 1), case["chunk"] + 7 * i) for i in range(case["chunks"])]).double()
        rad = _Radial(L, M, 1500.0, False, float(pts[:, 0].max()))
        cm, sm = _phases(pts[:, 2], L)
        _, c = _direct(pts[:, 0].contiguous(), torch.cos(pts[:, 1]), cm, sm, None, L, rad, _norm(1500.0, pts.shape[0]))
        return {"k_ln": rad.k, "c_ln": c}
    if f == "ingest":
        rec = _records(g, case)
        rec = rec.float().double() if case["f32"] else rec
        p = _spherical(rec) if case["cartesian"] else rec
        keep = p[:, 0] < 1500.0
        if case["nside"]:
            ring, j = _ring_pixels(case["nside"], p[:, 1], p[:, 2])
            keep &= _band_mask(case["nside"])[_ring_geometry(case["nside"])[3][ring] + j] == 1
        return p[keep].cpu().numpy()
    # integrals: w is linear between its nodes, so one rule per table segment serves every pair
    l, r, nk, nodes = case["l"], case["rmax"], case["nk"], case["nodes"]
    a = 0.3 + 0.2 * float(_uni(g, 1).cpu())
    xs = np.arange(nodes) * (r / (nodes - 1))
    wt = np.exp(-(xs / (a * r)) ** 2) * xs ** 2
    k = _zeros(l + 1, max(nk, 2))[l, :nk] / r
    gx, gw = np.polynomial.legendre.leggauss(10)
    h = r / (nodes - 1)
    x = (xs[:-1, None] + 0.5 * h * (gx + 1.0)).reshape(-1)
    t = 0.5 * (gx + 1.0)
    q = ((wt[:-1, None] + (wt[1:] - wt[:-1])[:, None] * t) * (0.5 * h * gw)).reshape(-1)
    xd = torch.from_numpy(x).cuda()
    jm = torch.stack([_jl_table(l + 1, float(v) * xd, only=l) for v in k])
    return ((jm * torch.from_numpy(q).cuda()) @ jm.T).cpu().numpy()
