// integrals.cu -- batched double spherical-Bessel integrals (the shot-noise integrals
// of the SFB power spectrum):
//
//   I(k1, k2) = int_0^rmax w(r) j_l(k1 r) j_l(k2 r) dr      (sbessel_integrator.cpp:53-110)
//
// The reference integrates pair by pair with GSL's adaptive Gauss-Kronrod (QAG, 21-point rule,
// epsrel 1e-7) over the sub-intervals between consecutive zeros of j_l(k1 r) and, inside
// each, of j_l(k2 r) (SBesselIntegrationRangeGenerator, :113-133), stopping once an outer
// interval adds less than 1e-10 of the total.  Here all pairs of a call share one quadrature:
// w is a FunctionInterpolator table (FunctionInterpolator.cpp:6-30), linear between its nodes, so
// the breakpoints are the table's nodes, and a fixed Gauss-Legendre rule per segment integrates the
// product of the two Bessel functions -- an entire function of exponential type k1 + k2 -- to
// 2^(2p+1) p!^4 / ((2p+1) (2p)!^3) (kappa / 2)^(2p), kappa = (k1 + k2) length: below 1e-14 for p = 2, 3, 4, 8 points
// and kappa up to 0.002, 0.046, 0.23, 3.4 (longer segments are cut).  kappa takes the largest k of pairs whose
// segments are cut into like numbers (within a factor of eight), and at least (l + 1) / rmax, the growth of j_l below
// its turning point.
//   k_dsb_nodes   abscissae and weights (rule times w) of a chunk of the quadrature
//   k_dsb_bessel  j_l(k x) for the call's distinct k: K x nodes evaluations instead of two per pair and node
//                 (a matrix of n x n pairs has n distinct k) -- the FP64 recurrences bound the call
//   k_dsb_pairs   a CTA per pair: the weighted product of two rows, added in a fixed order
// Measured, GB300: l 16, 32 x 32 pairs, 10001 nodes, host arrays in and out: 58.2 ms one warp per pair with
// both j_l evaluated at every node, 0.54 ms so.
#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "special.cuh"

namespace catana_gpu {

namespace {

constexpr int DSB_MAXP = 8;

struct DsbRule {
    double x[DSB_MAXP], w[DSB_MAXP];  // on [-1, 1]
    int p, cuts;                      // points per piece, pieces per table segment
    int64_t seg0, nseg;               // table segments [seg0, seg0 + nseg) meet (0, rmax)
    double wmin, wdx, wdxinv, rmax;
};

// node q = (segment, piece, point)
__global__ void k_dsb_nodes(DsbRule R, const double *__restrict__ wt, int64_t q0, int64_t nq, double *__restrict__ xo,
                            double *__restrict__ wo) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nq) return;
    const int64_t q = q0 + i, piece = q / R.p, sg = R.seg0 + piece / R.cuts;
    const int j = (int)(q - piece * R.p), c = (int)(piece % R.cuts);
    const double sa = fmax(0.0, R.wmin + (double)sg * R.wdx), sb = fmin(R.rmax, R.wmin + (double)(sg + 1) * R.wdx);
    const double len = (sb - sa) / R.cuts, half = 0.5 * len, x = sa + (double)c * len + half * (R.x[j] + 1.0);
    const double f = (x - R.wmin) * R.wdxinv - (double)sg;  // place in the table segment
    xo[i] = x;
    wo[i] = sb > sa ? R.w[j] * half * (wt[sg] + (wt[sg + 1] - wt[sg]) * f) : 0.0;
}

// a row of j_l(k x) per k, and the same times the weights: a pair is then one FP64 operation a node instead of two
// (1024 pairs of 32 k, 30k nodes: 124 -> 74 us)
__global__ void k_dsb_bessel(const double *__restrict__ k, const double *__restrict__ x, const double *__restrict__ w,
                             int64_t nq, int l, double *__restrict__ o, double *__restrict__ ow) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nq) return;
    const double j = jl_direct(l, k[blockIdx.y] * x[i]);
    o[(size_t)blockIdx.y * nq + i] = j;
    ow[(size_t)blockIdx.y * nq + i] = w[i] * j;
}

constexpr int DSB_T = 128;

// out[p] (+)= sum_q W[i1][q] J[i2][q], W = w J; first = 0 adds to the chunks before
__global__ void __launch_bounds__(DSB_T) k_dsb_pairs(const double *__restrict__ J, const double *__restrict__ W,
                                                     int64_t nq, const uint32_t *__restrict__ i1,
                                                     const uint32_t *__restrict__ i2, int first,
                                                     double *__restrict__ out) {
    __shared__ double s[DSB_T / 32];
    const int64_t p = blockIdx.x;
    // the smaller index first: I(k1, k2) and I(k2, k1) are the same sum
    const uint32_t a = min(i1[p], i2[p]), b = max(i1[p], i2[p]);
    const double *wa = W + (size_t)a * nq, *jb = J + (size_t)b * nq;
    double acc = 0.0;
#pragma unroll 4
    for (int64_t q = threadIdx.x; q < nq; q += DSB_T) acc = fma(wa[q], jb[q], acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < DSB_T / 32; ++k) acc += s[k];
        out[p] = first ? acc : out[p] + acc;
    }
}

// Gauss-Legendre nodes and weights on [-1, 1] (Newton on P_n from the asymptotic guesses
// cos(pi (i - 1/4) / (n + 1/2)); Abramowitz & Stegun 25.4.29)
void gauss_legendre(int n, double *x, double *w) {
    for (int i = 0; i < (n + 1) / 2; ++i) {
        double z = std::cos(kPi * (i + 0.75) / (n + 0.5)), pp = 0.0;
        for (int it = 0; it < 100; ++it) {
            double p1 = 1.0, p2 = 0.0;
            for (int j = 1; j <= n; ++j) {
                const double p3 = p2;
                p2 = p1;
                p1 = ((2.0 * j - 1.0) * z * p2 - (j - 1.0) * p3) / j;
            }
            pp = n * (z * p1 - p2) / (z * z - 1.0);
            const double dz = p1 / pp;
            z -= dz;
            if (std::fabs(dz) < 1e-16) break;
        }
        x[i] = -z;
        x[n - 1 - i] = z;
        w[i] = w[n - 1 - i] = 2.0 / ((1.0 - z * z) * pp * pp);
    }
}

// One call's weight table and range
struct DsbCall {
    int l;
    const double *w;
    int64_t wn;
    double wmin, wdx, rmax;
    // (k1 + k2) length of a piece of the segments inside (0, rmax), uncut
    double kappa(double kmax) const { return 2.0 * std::max(kmax, (l + 1.0) / rmax) * std::min(wdx, rmax); }
    double cuts(double kmax) const { return std::max(1.0, std::ceil(kappa(kmax) / 3.4)); }
};

// distinct k of a pass: their Bessel rows and the weighted ones, of 1024 nodes, take 512 MB
constexpr size_t DSB_MAXK = 31250;

// The integrals of pairs with k <= kmax (host arrays), by one rule
catana_status_t dsb_group(DeviceContext *ctx, const DsbCall &C, double kmax, const double *k1, const double *k2,
                          int64_t npairs, const std::vector<double> &ks, double *out, cudaStream_t st) {
    // each pair's two places among the distinct k
    std::vector<uint32_t> idx(2 * (size_t)npairs);
    for (int64_t i = 0; i < npairs; ++i) {
        idx[i] = (uint32_t)(std::lower_bound(ks.begin(), ks.end(), k1[i]) - ks.begin());
        idx[npairs + i] = (uint32_t)(std::lower_bound(ks.begin(), ks.end(), k2[i]) - ks.begin());
    }
    const size_t nk = ks.size();
    // the rule: table segments from that of 0 to that of r_max
    DsbRule R;
    R.wmin = C.wmin;
    R.wdx = C.wdx;
    R.wdxinv = 1.0 / R.wdx;
    R.rmax = C.rmax;
    R.seg0 = std::min<int64_t>(C.wn - 2, std::max<int64_t>(0, (int64_t)std::floor((0.0 - C.wmin) * R.wdxinv)));
    const int64_t sl = std::min<int64_t>(C.wn - 2, (int64_t)std::floor((C.rmax - C.wmin) * R.wdxinv));
    R.nseg = std::max<int64_t>(1, sl - R.seg0 + 1);
    const double kappa = C.kappa(kmax), cuts = C.cuts(kmax);
    R.p = kappa <= 0.002 ? 2 : kappa <= 0.046 ? 3 : kappa <= 0.23 ? 4 : 8;
    if (cuts * (double)R.nseg * R.p > 1e11) {
        set_error("sbessel_integrals: k r_max too large");
        return CATANA_ERR_ARG;
    }
    R.cuts = (int)cuts;
    gauss_legendre(R.p, R.x, R.w);
    const int64_t nodes = R.nseg * R.cuts * R.p;
    auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
    // nodes per pass: the Bessel rows and the weighted ones stay under 512 MB (up to DSB_MAXK distinct k)
    const int64_t chunk = std::max<int64_t>(1024, std::min<int64_t>(nodes, (int64_t)(512e6 / (16.0 * (double)nk))));
    const size_t wb = al((size_t)C.wn * 8), kb = al(nk * 8), ib = al((size_t)npairs * 8), ob = al((size_t)npairs * 8),
                 cb = al((size_t)chunk * 8), jb = al(nk * (size_t)chunk * 8);
    CG_CUDA_TRY(ctx->io_points.ensure(wb + kb + ib + ob + 2 * cb + 2 * jb + 256));
    char *d = ctx->io_points.as<char>();
    double *wd = reinterpret_cast<double *>(d), *kd = reinterpret_cast<double *>(d + wb),
           *od = reinterpret_cast<double *>(d + wb + kb + ib), *xd = reinterpret_cast<double *>(d + wb + kb + ib + ob),
           *qd = reinterpret_cast<double *>(d + wb + kb + ib + ob + cb),
           *jd = reinterpret_cast<double *>(d + wb + kb + ib + ob + 2 * cb),
           *jw = reinterpret_cast<double *>(d + wb + kb + ib + ob + 2 * cb + jb);
    uint32_t *id = reinterpret_cast<uint32_t *>(d + wb + kb);
    CG_CUDA_TRY(cudaMemcpyAsync(wd, C.w, (size_t)C.wn * 8, cudaMemcpyHostToDevice, st));
    CG_CUDA_TRY(cudaMemcpyAsync(kd, ks.data(), nk * 8, cudaMemcpyHostToDevice, st));
    CG_CUDA_TRY(cudaMemcpyAsync(id, idx.data(), idx.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, st));
    for (int64_t q0 = 0; q0 < nodes; q0 += chunk) {
        const int64_t nq = std::min(chunk, nodes - q0);
        k_dsb_nodes<<<ceil_div(nq, 256), 256, 0, st>>>(R, wd, q0, nq, xd, qd);
        k_dsb_bessel<<<dim3(ceil_div(nq, 256), (unsigned)nk), 256, 0, st>>>(kd, xd, qd, nq, C.l, jd, jw);
        k_dsb_pairs<<<(unsigned)npairs, DSB_T, 0, st>>>(jd, jw, nq, id, id + npairs, q0 == 0 ? 1 : 0, od);
        count_launch(3);
        CG_CUDA_TRY(cudaGetLastError());
    }
    CG_CUDA_TRY(cudaMemcpyAsync(out, od, (size_t)npairs * 8, cudaMemcpyDeviceToHost, st));
    CG_CUDA_TRY(cudaStreamSynchronize(st));
    return CATANA_OK;
}

// The same for any number of distinct k: in runs of pairs where they are too many for a pass
catana_status_t dsb_pairs(DeviceContext *ctx, const DsbCall &C, double kmax, const double *k1, const double *k2,
                          int64_t npairs, double *out, cudaStream_t st) {
    auto distinct = [&](int64_t b, int64_t e) {
        std::vector<double> ks(k1 + b, k1 + e);
        ks.insert(ks.end(), k2 + b, k2 + e);
        std::sort(ks.begin(), ks.end());
        ks.erase(std::unique(ks.begin(), ks.end()), ks.end());
        return ks;
    };
    std::vector<double> ks = distinct(0, npairs);
    if (ks.size() <= DSB_MAXK) return dsb_group(ctx, C, kmax, k1, k2, npairs, ks, out, st);
    const int64_t run = DSB_MAXK / 2;
    for (int64_t b = 0; b < npairs; b += run) {
        const int64_t e = std::min(npairs, b + run);
        const catana_status_t s = dsb_group(ctx, C, kmax, k1 + b, k2 + b, e - b, distinct(b, e), out + b, st);
        if (s != CATANA_OK) return s;
    }
    return CATANA_OK;
}

}  // namespace

}  // namespace catana_gpu

using namespace catana_gpu;

extern "C" {

catana_status_t catana_gpu_sbessel_integrals(const double *w_table, int64_t w_n, double w_min, double w_max,
                                             uint32_t l, double r_max, const double *k1, const double *k2,
                                             int64_t npairs, double *out, catana_gpu_stream_t stream) {
    if (!w_table || w_n < 2 || !(w_max > w_min) || !(r_max > 0.0) || !std::isfinite(r_max) || npairs < 0 ||
        (npairs > 0 && (!k1 || !k2 || !out))) {
        set_error("sbessel_integrals: need a w table of >= 2 nodes on w_min < w_max, r_max > 0, k1/k2/out");
        return CATANA_ERR_ARG;
    }
    if (npairs == 0) return CATANA_OK;
    double kmax = 0.0;
    for (int64_t i = 0; i < npairs; ++i) {
        if (!(k1[i] >= 0.0) || !(k2[i] >= 0.0) || !std::isfinite(k1[i]) || !std::isfinite(k2[i])) {
            set_error("sbessel_integrals: k1 and k2 must be >= 0 and finite");
            return CATANA_ERR_ARG;
        }
        kmax = std::max(kmax, std::max(k1[i], k2[i]));
    }
    if (w_min > 0.0 || r_max > w_max) {
        set_error("argument outside range for which this FunctionInterpolator is defined");
        return CATANA_ERR_DOMAIN;
    }
    int cs;
    DeviceContext *ctx = get_context(&cs);
    if (!ctx) return (catana_status_t)cs;
    std::lock_guard<std::mutex> g(ctx->mu);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    DsbCall C;
    C.l = (int)l;
    C.w = w_table;
    C.wn = w_n;
    C.wmin = w_min;
    C.wdx = (w_max - w_min) / (double)(w_n - 1);
    C.rmax = r_max;
    if (!(C.cuts(kmax) < 2e9)) {
        set_error("sbessel_integrals: k r_max too large");
        return CATANA_ERR_ARG;
    }
    if (C.cuts(kmax) < 8.0) return dsb_pairs(ctx, C, kmax, k1, k2, npairs, out, st);
    // The pairs by the octal order of their pieces per segment: a pair is not integrated on pieces that only a much
    // larger k of the call asks for.
    std::vector<int> order(npairs);
    int lo = INT_MAX, hi = 0;
    for (int64_t i = 0; i < npairs; ++i) {
        order[i] = (int)(std::log2(C.cuts(std::max(k1[i], k2[i]))) / 3.0);
        lo = std::min(lo, order[i]);
        hi = std::max(hi, order[i]);
    }
    if (lo == hi) return dsb_pairs(ctx, C, kmax, k1, k2, npairs, out, st);
    for (int o = lo; o <= hi; ++o) {
        std::vector<int64_t> at;
        std::vector<double> a, b;
        double km = 0.0;
        for (int64_t i = 0; i < npairs; ++i)
            if (order[i] == o) {
                at.push_back(i);
                a.push_back(k1[i]);
                b.push_back(k2[i]);
                km = std::max(km, std::max(k1[i], k2[i]));
            }
        if (at.empty()) continue;
        std::vector<double> v(at.size());
        const catana_status_t s = dsb_pairs(ctx, C, km, a.data(), b.data(), (int64_t)at.size(), v.data(), st);
        if (s != CATANA_OK) return s;
        for (size_t i = 0; i < at.size(); ++i) out[at[i]] = v[i];
    }
    return CATANA_OK;
}

}  // extern "C"
