// common.cuh -- shared declarations of the catana_gpu library (host side).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <cmath>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/catana_gpu.h"

namespace catana_gpu {

// Launch counter behind catana_gpu_launch_count().
extern std::atomic<uint64_t> g_launches;
inline void count_launch(uint64_t n = 1) { g_launches.fetch_add(n, std::memory_order_relaxed); }

void set_error(const std::string &msg);

// Kernel timing (catana_gpu_profile_*): prof_begin/prof_end bracket one launch of
// the dominant kernel when profiling is enabled.
void prof_begin(cudaStream_t st);
void prof_end(cudaStream_t st, double algo_flops);

// Test hook (catana_gpu_test_alloc_limit): larger buffers than this cannot be had by this thread's calls (0: no limit)
extern thread_local size_t t_alloc_limit;

// Grow-only device buffer, allocated a quarter larger than asked for where that can be had.  A failed ensure() leaves
// it empty, so whoever caches something in it forgets that before the call.
struct DevBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
    cudaError_t ensure(size_t need) {
        const bool refuse = t_alloc_limit && need > t_alloc_limit;
        if (need <= bytes && !refuse) return cudaSuccess;
        release();
        size_t cap = need + need / 4;
        cudaError_t e = refuse ? cudaErrorMemoryAllocation : cudaMalloc(&ptr, cap);
        if (e == cudaErrorMemoryAllocation && !refuse) {
            cudaGetLastError();
            e = cudaMalloc(&ptr, cap = need);
        }
        if (e == cudaSuccess) {
            bytes = cap;
        } else {
            ptr = nullptr;
            cudaGetLastError();  // reported here, not by the next launch
        }
        return e;
    }
    template <class T> T *as() const { return reinterpret_cast<T *>(ptr); }
    void release() {
        if (ptr) cudaFree(ptr);
        ptr = nullptr;
        bytes = 0;
    }
};

// Cached split-form tables (per device): j_l piecewise polynomials, recurrence
// coefficients and the largest |j_l| per l.
struct SplitCache {
    int lmax = -1, nmax = -1, nint = -1;
    std::vector<double> maxj;   // 1.05 max |j_l| (first maximum)
    std::vector<double> zpeak;  // where that maximum sits (j_l rises monotonically below)
};

// Per-device state: workspace and cached tables.  Guarded by `mu`.
struct DeviceContext {
    std::mutex mu;
    int device = 0;
    int sm_count = 0;
    int cc_major = 0, cc_minor = 0;
    // workspace
    DevBuf soa;        // point SoA (r, x, w, cos phi, sin phi, phase fraction) of the current chunk
    DevBuf state;      // Legendre recurrence rows
    DevBuf partial;    // per-slab partial sums
    DevBuf flmn;       // f_lmn accumulator (complex, packed)
    DevBuf kln;        // k_ln on device
    DevBuf coef;       // Legendre recurrence coefficients
    DevBuf tables;     // j_l interpolation tables (FP64 lerp)
    DevBuf misc;       // error word, small scalars (never grown past 256 bytes: callers hold pointers into it)
    DevBuf cat_scratch;  // per-catalog scalars of batched runs (extents, weight sums)
    DevBuf io_points;  // staging of host inputs
    DevBuf io_out;     // staging of outputs
    DevBuf split_ws;   // split-form workspace
    DevBuf split_tab;  // split-form tables
    DevBuf split_plan; // split-form plan (catalog descriptors, items, reductions)
    SplitCache split_cache;
    std::map<std::string, std::pair<double, int>> split_tuned;  // autotuned (waves, m-block cap) per catalog set
    double split_last_waves = 0.0;
    int split_last_mblk = 0;
    cudaStream_t capture_stream = nullptr;      // stream the split level loop is captured on
    cudaEvent_t ws_event = nullptr;             // end of the last call's work (WsOrder)
    DevBuf hp_ws;      // HEALPix workspace
    DevBuf ingest_ws;  // ingest: converted records, keep flags, block counts, window, mask
    // kernels whose shared-memory limit this device's context has raised (the
    // attribute is per device, so it is tracked here rather than per process)
    bool attr_fp64 = false, attr_split = false, attr_healpix = false;
    // cache keys
    int coef_lmax = -1;
    int tab_lmax = -1, tab_nmax = -1;
    std::vector<double> tab_dxinv, tab_zmax;  // per l
    DevBuf poly;       // piecewise FP64 j_l polynomials [l][interval][12] (CATANA_JL_POLY)
    int poly_lmax = -1, poly_nint = -1;
    // plain path on the tensor cores (plain_tc.cu)
    DevBuf tc_ws;      // sort scratch, point records, Legendre rows, phase tables
    DevBuf tc_coef;    // (beta, A) of the monic recurrence
    DevBuf tc_tab;     // (y0 - dy, dy) lerp tables, dx^-1 and z_max per l
    DevBuf tc_jarr;    // j_l arrays of the modes without a table
    DevBuf tc_poly;    // the polynomials of `poly` as integers
    int tc_poly_lmax = -1, tc_poly_nint = -1;
    int tc_coef_lmax = -1, tc_tab_lmax = -1, tc_tab_nmax = -1;
    size_t tc_tab_off = 0;
    bool attr_tc = false;
};

DeviceContext *get_context(int *status);

// The workspaces and the cached tables of a context serve every stream that computes on its device, and calls on
// device arrays return before their work is done.  An entry point holds one of these, under the context's mutex,
// from before it touches any of them -- a table that is built for another nmax overwrites the one that an earlier
// call still reads -- until all of its work is enqueued: its stream then waits for the work of the call before
// it, and the next one's for its own.
class WsOrder {
public:
    WsOrder(DeviceContext *ctx, cudaStream_t st);
    ~WsOrder();
    WsOrder(const WsOrder &) = delete;
    WsOrder &operator=(const WsOrder &) = delete;
    cudaError_t err;  // of the wait

private:
    DeviceContext *ctx_;
    cudaStream_t st_;
};

// Bessel zeros (host, cached): z[l][n] for n < count.  Thread-safe.
const double *zeros_for(unsigned l, int count);
// k_ln table row-major (lmax x nmax), host.
void kln_table(int lmax, int nmax, double rmax, double *out);

inline int ceil_div(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

#define CG_CUDA_TRY(expr)                                                                        \
    do {                                                                                         \
        cudaError_t _e = (expr);                                                                 \
        if (_e != cudaSuccess) {                                                                 \
            ::catana_gpu::set_error(std::string(#expr) + ": " + cudaGetErrorString(_e));         \
            return _e == cudaErrorMemoryAllocation ? CATANA_ERR_NOMEM : CATANA_ERR_CUDA;          \
        }                                                                                        \
    } while (0)

// j_l evaluation of the FP64 plain path: the reference's linear table, the direct
// evaluation, or the piecewise FP64 polynomials (CATANA_JL_POLY).
enum JlMode { JL_MODE_LERP = 0, JL_MODE_EXACT = 1, JL_MODE_POLY = 2 };

// The smallest and the largest |w| of a catalog that are neither 0 nor infinite nor NaN (none: lo > hi).
struct WeightRange {
    double lo = HUGE_VAL, hi = 0.0;
    void add(double w) {
        const double a = std::fabs(w);
        if (!(a > 0.0 && a < HUGE_VAL)) return;
        if (a < lo) lo = a;
        if (a > hi) hi = a;
    }
};

// Plain raw form (sfb_fp64.cu).  All pointers device.  Accumulates into f_acc (complex, packed by l,
// un-normalised); the caller normalises.  wr: of weights_dev, or null where the caller does not know it yet and will
// start again if plain_tc_holds() says no to it.
catana_status_t fp64_raw_accumulate(DeviceContext *ctx, const double *points_dev, const double *weights_dev,
                                    const WeightRange *wr, int64_t npoints, int lmax, int nmax, double rmax, JlMode jl,
                                    const double *kln_dev, double *f_acc_dev, int *err_dev, cudaStream_t st);
// The same sum with its contraction on the tensor cores (plain_tc.cu), where the device has them and
// lmax <= 512; with JL_MODE_POLY the caller has prepared ctx->poly and passes the largest radius (else rtop = 0).
bool plain_tc_takes(const DeviceContext *ctx, int lmax, int nmax, double rmax);
bool plain_tc_pays(int64_t npoints, int lmax, int nmax, JlMode jl);  // and whether it is the faster one
double plain_tc_blocks(int lmax, int nmax);  // blocks that a CTA of it walks
bool plain_tc_holds(const WeightRange &wr);  // and whether its fixed-point terms hold weights of this range
catana_status_t plain_tc_accumulate(DeviceContext *ctx, const double *points_dev, const double *weights_dev,
                                    int64_t npoints, int lmax, int nmax, double rmax, JlMode jl, double rtop,
                                    const double *kln_dev, double *f_acc_dev, int *err_dev, cudaStream_t st);
// f *= norm; c_ln from f (device).
catana_status_t finish_flmn_cln(double *f_dev, double norm, int lmax, int nmax, double *c_ln_dev,
                                cudaStream_t st);
// FP64 lerp tables (1000*nmax nodes per l) for l < lmax, cached in ctx->tables.
catana_status_t ensure_lerp_tables(DeviceContext *ctx, int lmax, int nmax, cudaStream_t st);
// Legendre coefficients for l < lmax, cached in ctx->coef.
catana_status_t ensure_coefs(DeviceContext *ctx, int lmax, cudaStream_t st);

// A catalog in RING pixels, with its ring tables (device pointers).
struct PixelCatalog {
    const double *r;            // radii grouped by pixel
    const int64_t *offs;        // [npix + 1]
    int64_t npix;
    int nrings;
    bool conj;                  // CATANA_HEALPIX_CONJ_FIX
    const int64_t *ring_start;
    const int *ring_pix;
    const double *ring_x, *ring_phi;
    const double2 *tw;          // e^{-2 pi i k / N} per ring length, at tw_off[ring]
    const int64_t *tw_off;
};
// The pixelized sum (un-normalised, times k_ln) as a sum over points at their pixels' centres.
catana_status_t plain_tc_pixels(DeviceContext *ctx, const PixelCatalog &pix, int64_t npoints, int lmax, int nmax,
                                double rmax, JlMode jl, const double *kln_dev, double *f_acc_dev, int *err_dev,
                                cudaStream_t st);

// One catalog of a split-form run (device pointers; f_acc zeroed by the caller).
struct SplitCatInput {
    const double *pts = nullptr;  // n x 3 (r, theta, phi)
    const double *w = nullptr;    // optional weights
    const float *pts32 = nullptr; // or: float32 records (r, theta, phi) and weights
    const float *w32 = nullptr;
    double max_r = -1.0, max_w = -1.0;  // >= 0: extents known to the caller (skips a read-back)
    int64_t n = 0;
    int lmax = 0, nmax = 0;
    double rmax = 1.0;
    double kmax = 0.0;            // > 0: keep only k_ln <= kmax
    double *kln_dev = nullptr;    // k_ln (lmax x nmax), already on the device
    double *f_acc = nullptr;      // packed complex f_lmn accumulator
    bool accurate = false;        // CATANA_SPLIT_ACCURATE: Reinsch-modified Legendre rows (always above lmax 256)
};
// Split form over several catalogs: level-synchronous launches over all of them,
// optionally captured as one CUDA graph.  `waves` = CTAs per SM each level's work
// items are cut for, `mblk` the most complex m per work item (128 or 64); waves <= 0
// autotunes both (timed sample levels, cached per catalog set).
catana_status_t split_run(DeviceContext *ctx, std::vector<SplitCatInput> &cats, bool use_graph, double waves,
                          int mblk, int *err_dev, cudaStream_t st);

// Convert, filter and compact n device records (ingest.cu); *n_out kept, in order.
catana_status_t ingest_dev(DeviceContext *ctx, const void *rec_dev, int64_t n, const catana_ingest_t &spec,
                           double *out_dev, int64_t *n_out, cudaStream_t st);

// Split (tensor-core) raw path (sfb_split.cu).
catana_status_t split_raw_accumulate(DeviceContext *ctx, const double *points_dev, const double *weights_dev,
                                     int64_t npoints, int lmax, int nmax, double rmax, const double *kln_dev,
                                     double *f_acc_dev, int *err_dev, cudaStream_t st, bool accurate);

// Stable radix sort of (key, index) pairs by the low key_bits bits (sort.cu); hist_scratch:
// radix_hist_words(n) words, which does not fall as n grows.
size_t radix_hist_words(int64_t n);
catana_status_t radix_sort_pairs(uint32_t *keys, uint32_t *vals, uint32_t *tmp_keys, uint32_t *tmp_vals, int64_t n,
                                 int key_bits, uint32_t *hist_scratch, cudaStream_t st);

// In-place exclusive scan of uint32 words (sort.cu).
catana_status_t scan_u32(uint32_t *data, int64_t count, cudaStream_t st);

// HEALPix (healpix.cu).
catana_status_t healpix_bin_dev(DeviceContext *ctx, int64_t nside, const double *points_dev, int64_t npoints,
                                int64_t *offsets_dev, double *r_sorted_dev, int *err_dev, cudaStream_t st);
catana_status_t healpix_ang2pix_dev(int64_t nside, const double *theta, const double *phi, int64_t n,
                                    int64_t *pix, int *err_dev, cudaStream_t st);
catana_status_t healpix_pix2ang_dev(int64_t nside, const int64_t *pix, int64_t n, double *theta, double *phi,
                                    cudaStream_t st);
// offsets_host, kln_host (L x M) and r_host: host copies of the offsets (the fullest pixel), of k_ln and of the radii
// (map levels that lie inside the j_l table skip the per-point range test).
catana_status_t healpix_sfb_dev(DeviceContext *ctx, int64_t nside, const int64_t *offsets_dev,
                                const double *r_sorted_dev, const int64_t *offsets_host, int64_t npoints, int lmax,
                                int nmax, double rmax, bool interpolated, bool conj_fix, const double *kln_dev, const double *kln_host,
                                const double *r_host, double norm, double *f_dev, double *c_ln_dev, int *err_dev,
                                cudaStream_t st);

}  // namespace catana_gpu
