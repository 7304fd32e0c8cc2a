// plain_tc.cu -- the plain (FP64-accurate) raw SFB sum with its contraction on the tcgen05
// tensor cores.
//
//   f_l(m, n) = k_ln sum_i w_i j_l(k_ln r_i) P_lm(cos theta_i) e^{-i m phi_i}   (sfb_raw.cpp:56-84)
//
// GB300 issues two FP64 FMAs per SM and cycle, so the FP64 contraction (k_fp64_raw_l,
// 2 nmax (l + 1) FMAs per point and l) leaves everything else idle.  Here both factors become
// fixed-point numbers cut into signed 8-bit digits, and the digit products run as FP16 MMAs whose
// FP32 accumulators hold exact integers:
//   J[n][i]    = j_l(k_ln r_i) 2^(63 - EJ_n)                             -> digits J_0 .. J_7
//   Y[m,ri][i] = w_i P_lm(x_i) (cos, -sin)(m phi_i) 2^(55 - EP_m - EW)   -> digits Y_0 .. Y_6
//   D_d = sum_{a + b = d} Y_a J_b^T,  d = 0 .. 7   (35 digit products)
// A digit is in [-128, 127], so a D_d entry of 128 points is at most 7 * 128 * 2^14 < 2^24: every
// FP32 sum is exact.  After 128 points the eight D_d are added, as integers with weights
// 256^(7 - d), to one 64-bit register per (m, ri, n), which holds the slab's whole sum.
// What is rounded: the operands (Y to 2^-55 of its row's bound, J to 2^-63), the products of digits
// a + b > 7 (2^-64), and each group's sum (2^-54 of the slab's largest term).  (With seven digits of J,
// 28 products, the sums erred by 30% more, at the same speed.)  The rows' bounds are kept close to
// the values: points are sorted by radius, a CTA owns a contiguous slab of at most 2048 of them, EJ
// bounds |j_l| over the slab's radii (Debye's and Watson's inequalities), EP bounds
// |P_lm| over the slab's points from the two levels before, EW the slab's weights.
//
// What a point costs besides the MMAs (CUDA cores):
//   * P_lm: the monic recurrence Q_l = x Q_{l-1} - beta_lm Q_{l-2} (P_lm = A_lm Q_lm, A_lm applied
//     at the slab's end) in FP64, two operations per (point, m);
//   * the phase e^{-i m phi} w as a 58-bit table per (point, m), written once per call;
//     Y = the upper half of a 64 x 64-bit integer product;
//   * j_l from the reference's linear table (SBesselInterpolator.cpp:10-26): the table position
//     k r / dx is a 64 x 64-bit integer product, the interpolation one FP64 FMA on (y0 - dy, dy);
//     or, in the other j_l modes and for pixelized catalogs, read from an array that another kernel filled.
// FP64 work: 3 operations per (point, m) and (point, n) instead of 2 nmax (l + 1).
//
// Schedule: one CTA per slab walks every level of the launch (its Legendre rows are its own, so
// levels need no grid-wide wait), 64 complex m x up to 64 radial orders at a time.  Warps 0..10
// write the digits of 32-point tiles into two shared-memory buffers (units of four m or eight
// radial orders, dealt round robin across tiles), warp 11 issues the MMAs (all digits J_0 .. J_{7-a}
// of B in one N <= 256 instruction, since D_{a + b} lie side by side), warps 12..19 fold.  D lies in
// two regions, so that MMAs run while sums are folded: with at most 32 radial orders they take the
// groups in turn (each folded by all eight warps), otherwise the radial orders below and from 32
// (each folded by four warps).  Slab sums go to HBM as FP64 and are added in slab
// order (k_ptc_reduce): results do not depend on timing.
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "special.cuh"
#include "tc05.cuh"

namespace catana_gpu {

namespace {

constexpr int TC_KT = 32;        // points per tile (two K = 16 MMA steps)
constexpr int TC_GROUP = 4;      // tiles per exact FP32 sum (128 points)
constexpr int TC_DY = 7;         // 8-bit digits of Y
constexpr int TC_DG = 8;         // 8-bit digits of J, digit sums
constexpr int TC_MB = 64;        // complex m per block (128 MMA rows)
constexpr int TC_NB = 64;        // most radial orders per block
constexpr int TC_OPW = 11;       // operand warps
constexpr int TC_OPT = 32 * TC_OPW;
constexpr int TC_FOLD0 = 12;     // first fold warp (warp 11 issues the MMAs)
constexpr int TC_THREADS = 640;  // 12 + 8 warps
constexpr int TC_SLAB_TILES = 64;  // most tiles per slab (an exact sum's count has room for 240)
constexpr int TC_LMAX = 512;     // |Q_lm| and A_lm stay inside FP64 up to here
constexpr uint64_t TC_WAIT_NS = 1000000000ull;
constexpr uint64_t TC_OFF_Y = 0x0080808080808080ull;  // 128 in every digit
constexpr uint64_t TC_OFF_J = 0x8080808080808080ull;
constexpr int TC_NH = 32;        // radial orders per D region
constexpr uint32_t TC_DREG = TC_DG * TC_NH;  // columns of a D region

// shared memory from a 1024-aligned base: two operand buffers, then the block tables
constexpr uint32_t TC_YD = 8192;                       // one Y digit: 4 k-groups x 2 atoms of 1 KB
constexpr uint32_t TC_SY = TC_DY * TC_YD;
constexpr uint32_t TC_SJ = 8 * 4 * 1024;               // J digits: 4 k-groups x up to 2 x 4 atoms
constexpr uint32_t TC_BUF = TC_SY + TC_SJ;
constexpr uint32_t TC_RING = 8;                        // block tables in flight (the fold may be five blocks behind)
constexpr uint32_t TC_OFF_N = 2 * TC_BUF;              // uint4 per n: (kd hi, kd lo, shift, EJ)
constexpr uint32_t TC_OFF_M = TC_OFF_N + TC_RING * TC_NB * 16;  // per m: (beta, EP)
constexpr uint32_t TC_OFF_MX = TC_OFF_M + TC_RING * TC_MB * 16; // max |Q| (upper words), three levels
constexpr uint32_t TC_SMEM = TC_OFF_MX + 3 * TC_LMAX * 4 + 1024;
static_assert(TC_SMEM <= 232448 - 1024, "k_ptc_main shared memory");

struct TcSlab {
    double rmin, rmax;  // of |r|
    int ew;             // |w| < 2^ew
    int ec;             // at most 2^ec points in an entry of a pixelized catalog (0 otherwise)
};

// One call's words on the device, zero at first
struct TcCall {
    int poison;  // TC_POISON_*
    int etop;    // 2048 + the largest EW of its slabs so far
    unsigned long long count;  // a pixelized catalog's entries
};

// 2^e in two factors that are normal numbers, |e| <= 2000
__device__ __forceinline__ double pow2_lo(int e) { return __hiloint2double((1023 + (e >> 1)) << 20, 0); }
__device__ __forceinline__ double pow2_hi(int e) { return __hiloint2double((1023 + e - (e >> 1)) << 20, 0); }

struct TcArgs {
    int l0, l1;                 // levels of the launch
    int nmax, lmp;              // radial orders; row pitch in m (lmax rounded up to 4)
    int tiles, tslab;           // tiles of the chunk, tiles per slab
    const ulonglong2 *phase;    // [tile][lmp][32]: w cos, -w sin of m phi, times 2^(58 - EW), words split at
                                // 2^32 into two signed halves
    double *rows;               // [2][tile][lmp][32]: Q_l by the parity of l
    const uint64_t *rint;       // [point]: r 2^(62 - er)
    const double2 *xs;          // [point]: cos theta, sin theta
    const TcSlab *slab;
    const double2 *coef;        // (beta, A) per (l, m)
    const uint4 *ntab;          // [slab][l - l0][n]: (kd hi, kd lo, shift, EJ)
    const double2 *tab;         // lerp tables [l][npts]: (y_i - dy_i, dy_i), or null
    int npts;
    const uint64_t *jarr;       // J with its digit offset, [l - l0][tile][nmax][32], where tab is null
    uint32_t *maxq;             // [slab][3][TC_LMAX]: level maxima between launches
    double *partial;            // [slab][l - l0][n][2 (l + 1)]
    int64_t pslab;              // doubles per slab in partial
    uint64_t wait_ns;           // limit of every wait
    int stall;                  // test hook: the MMAs wait for a hand-off that nothing makes
    const TcCall *call;
    int *err;
};

__device__ __forceinline__ uint64_t shr64(uint64_t v, int s) {  // 0 past 63
    uint64_t r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    return r;
}

// x as upper and lower words that are both signed: x = hi 2^32 + lo
__device__ __forceinline__ uint64_t signed_halves(int64_t x) { return (uint64_t)x + ((uint64_t)(x & 0x80000000ll) << 1); }

// Byte `byte` of eight consecutive rows' or columns' values at one point as FP16 digits, 16 bytes:
// 0x6400 | b is 1024 + b, minus 1152 is b - 128.
template <int BYTE>
__device__ __forceinline__ void store_digit(uint8_t *p, const uint64_t (&u)[8]) {
    const __half2 c = __half2half2(__ushort_as_half(0x6480));  // 1152
    constexpr uint32_t b = BYTE & 3;
    uint32_t w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const uint32_t x = BYTE >= 4 ? (uint32_t)(u[2 * k] >> 32) : (uint32_t)u[2 * k];
        const uint32_t y = BYTE >= 4 ? (uint32_t)(u[2 * k + 1] >> 32) : (uint32_t)u[2 * k + 1];
        uint32_t t = __byte_perm(x, y, b | (b << 4) | ((4 + b) << 8) | ((4 + b) << 12));
        t = (t & 0x00ff00ffu) | 0x64006400u;
        const __half2 h = __hsub2(*reinterpret_cast<__half2 *>(&t), c);
        w[k] = *reinterpret_cast<const uint32_t *>(&h);
    }
    *reinterpret_cast<uint4 *>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}
template <int A, int N>
struct Digits {
    template <class F>
    static __device__ __forceinline__ void each(F &&at, const uint64_t (&u)[8]) {  // digit A of N at at(A)
        store_digit<N - 1 - A>(at(A), u);
        if constexpr (A + 1 < N) Digits<A + 1, N>::each(at, u);
    }
};

// FP64 load where pred holds, 0 elsewhere (rows that this kernel also writes)
__device__ __forceinline__ double ld_if(const double *p, bool pred) {
    double v;
    asm volatile("{\n.reg .pred q;\nsetp.ne.s32 q, %2, 0;\nmov.f64 %0, 0d0000000000000000;\n"
                 "@q ld.global.L1::no_allocate.f64 %0, [%1];\n}"
                 : "=d"(v)
                 : "l"(p), "r"((int)pred)
                 : "memory");
    return v;
}

// the same for a pair of read-only words; L1 is left to the j_l table
__device__ __forceinline__ ulonglong2 ld_if(const ulonglong2 *p, bool pred) {
    ulonglong2 v;
    asm volatile("{\n.reg .pred q;\nsetp.ne.s32 q, %3, 0;\nmov.u64 %0, 0;\nmov.u64 %1, 0;\n"
                 "@q ld.global.nc.L1::no_allocate.v2.u64 {%0, %1}, [%2];\n}"
                 : "=l"(v.x), "=l"(v.y)
                 : "l"(p), "r"((int)pred));
    return v;
}

// j 2^(63 - EJ) with the digit offset; w = (EJ + 1022) 2^20
__device__ __forceinline__ uint64_t j_digits(double j, uint32_t w) {
    const uint32_t jh = (uint32_t)__double2hiint(j), jl = (uint32_t)__double2loint(j);
    const int s = (int)(w - (jh & 0x7ff00000u)) >> 20;
    const uint64_t p = shr64(((uint64_t)((jh & 0xfffffu) | 0x100000u) << 42) | ((uint64_t)jl << 10), s);
    return jh >> 31 ? TC_OFF_J - p : TC_OFF_J + p;
}

// The position of k r in the linear tables from a radius and an entry of k_ptc_ntab: node and FP64 fraction
__device__ __forceinline__ uint32_t lerp_at(uint64_t r, const uint4 &kd, int npts, double &f) {
    const uint32_t rh = (uint32_t)(r >> 32), rl = (uint32_t)r;
    const uint64_t tt = (uint64_t)rl * kd.x + (uint64_t)rh * kd.y;
    const uint64_t res = (uint64_t)rh * kd.x + (tt >> 32);
    const uint32_t fh = __funnelshift_l((uint32_t)res, (uint32_t)(res >> 32), kd.z);
    const uint32_t fl = __funnelshift_l((uint32_t)tt, (uint32_t)res, kd.z);
    f = __hiloint2double((int)(0x3ff00000u | (fh >> 12)), (int)__funnelshift_l(fl, fh, 20));
    return min((uint32_t)(res >> 32) >> (32u - kd.z), (uint32_t)(npts - 1));
}

// log2 of a bound on |j_l| over [z1, z2] (FP32; checked to exceed log2 |j_l| up to 1e-6 for every l < 512):
// below l + 1/2 Debye's inequality at z2, beyond it Watson's M^2 < 2 / (pi sqrt(z^2 - nu^2)) at z1, never
// more than the maximum of j_l, 0.89 (l + 1/2)^(-5/6)
__device__ __forceinline__ float jl_log2_bound(int l, float z1, float z2) {
    const float nu = (float)l + 0.5f;
    const float mx = fminf(0.f, -0.1681228f - 0.8333333f * log2f(nu));
    float b = mx;
    if (z2 < nu) {
        const float z = fmaxf(z2, 1e-30f);
        const float s = sqrtf((nu - z) * (nu + z));
        b = (s - nu * logf((nu + s) / z)) * 1.4426950f - 1.f - 0.5f * log2f(z) - 0.5f * log2f(s);
    } else if (z1 > nu) {
        b = -0.5f * log2f(z1) - 0.25f * log2f((z1 - nu) * (z1 + nu));
    }
    return fminf(b, mx);
}

__device__ __forceinline__ void op_bar() { asm volatile("barrier.sync 2, 352;" ::: "memory"); }
__device__ __forceinline__ void tc_arrive(uint64_t *mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc05::smem_u32(mbar)) : "memory");
}
__device__ __forceinline__ void tmem_ld2(uint32_t taddr, uint32_t (&v)[2]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(v[0]), "=r"(v[1]) : "r"(taddr));
}

// Block (l, m-block, n-block) sequence of the launch, walked alike by the operand and the fold warps.
struct TcBlock {
    int l, mb0, mcount, n0, ncount;
    int nb0, nb1;  // columns per digit (multiples of 16) of the radial orders below TC_NH and from it
};
template <class F>
__device__ __forceinline__ void tc_blocks(const TcArgs &a, F &&body) {
    int seq = 0;
    for (int l = a.l0; l < a.l1; ++l)
        for (int mb0 = 0; mb0 <= l; mb0 += TC_MB)
            for (int n0 = 0; n0 < a.nmax; n0 += TC_NB) {
                TcBlock b;
                b.l = l;
                b.mb0 = mb0;
                b.mcount = min(TC_MB, l + 1 - mb0);
                b.n0 = n0;
                b.ncount = min(TC_NB, a.nmax - n0);
                b.nb0 = min(TC_NH, (b.ncount + 15) & ~15);
                b.nb1 = max(0, ((b.ncount + 15) & ~15) - TC_NH);
                body(b, seq++);
            }
}

// What bounds it: the operand warps' dependent instructions.  A unit (4 complex m or 8 radial orders at 32
// points) is ~450 instructions of one warp and takes it 4.5k cycles, with eleven such warps an SM; measured on
// 200k points, lmax 96, nmax 48 (ncu): 1.57 instructions a cycle, FP64 pipe 32%, ALU 40%, tensor pipe 26%, DRAM
// 13.8 + 3.7 GB; 20 ms against 281 with FP64 FMAs on CUDA cores.  More operand warps spill at the registers that
// are left (15 of them: +25%), fewer are slower, and J from a kernel of its own (which takes 60% off the units of
// n) made it 22.7 ms.
template <bool LERP>
__global__ void __launch_bounds__(TC_THREADS, 1) k_ptc_main(TcArgs a) {
    extern __shared__ uint8_t tc_smem[];
    uint8_t *sm = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(tc_smem) + 1023) & ~uintptr_t(1023));
    __shared__ uint64_t full[2], empty[2], gdone[2], dfree[2], drain;
    __shared__ uint32_t tmem_sh;
    __shared__ int abort_sh;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int slab = blockIdx.x;
    const int t0 = slab * a.tslab, t1 = min(a.tiles, t0 + a.tslab);
    const bool alt = a.nmax <= TC_NH;  // the D regions take the groups in turn
    constexpr uint32_t tcols = 512;
    uint4 *s_n = reinterpret_cast<uint4 *>(sm + TC_OFF_N);
    double2 *s_m = reinterpret_cast<double2 *>(sm + TC_OFF_M);  // (beta, EP as int bits)
    uint32_t *s_mx = reinterpret_cast<uint32_t *>(sm + TC_OFF_MX);
    volatile int *abort_v = &abort_sh;
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            tc05::mbar_init(&full[b], TC_OPW);
            tc05::mbar_init(&empty[b], 1);
            tc05::mbar_init(&gdone[b], 1);
            tc05::mbar_init(&dfree[b], alt ? 256 : 128);
        }
        tc05::mbar_init(&drain, 1);
        abort_sh = 0;
    }
    // level maxima carried over from the launch before (levels l0 - 1, l0 - 2)
    for (int k = tid; k < 3 * TC_LMAX; k += TC_THREADS)
        s_mx[k] = a.l0 > 0 ? a.maxq[(size_t)slab * 3 * TC_LMAX + k] : 0u;
    if (warp == TC_FOLD0) tc05::tmem_alloc(&tmem_sh, tcols);
    tc05::fence_before();
    __syncthreads();
    tc05::fence_after();
    const uint32_t tmem = tmem_sh;
    // a bounded wait; once one ran out every later wait of the warp returns at once, those of the others once
    // they have to wait at all, and the roles walk on to their ends.  Each warp whose wait ran out reports it.
    auto wait = [&](uint64_t *bar, uint32_t parity, bool &dead) {
        if (dead || __all_sync(0xffffffffu, tc05::mbar_try(bar, parity))) return;
        dead = __any_sync(0xffffffffu, *abort_v || !tc05::mbar_wait(bar, parity, a.wait_ns));
        if (dead) *abort_v = 1;
    };

    if (warp < TC_OPW) {
        uint32_t use = 0;  // tiles written so far
        int ofs = 0;       // units dealt so far, mod TC_OPW
        bool dead = false;
        const uint32_t lk = (uint32_t)(lane >> 3), lr = (uint32_t)(lane & 7);  // K row of this point: group, row
        const size_t lset = (size_t)a.tiles * a.lmp * TC_KT;
        tc_blocks(a, [&](const TcBlock &b, int seq) {
            const int l = b.l;
            const int ring = seq & (int)(TC_RING - 1);
            uint4 *tn = s_n + ring * TC_NB;
            double2 *tm = s_m + ring * TC_MB;
            // past the count: zero digits
            uint4 e = make_uint4(0u, 0u, 31u, 2022u << 20);
            double beta = 0.0;
            if (tid < b.ncount) e = a.ntab[((size_t)slab * (a.l1 - a.l0) + (l - a.l0)) * a.nmax + b.n0 + tid];
            if (tid >= 64 && tid < 64 + b.mcount) beta = a.coef[(size_t)l * (l + 1) / 2 + b.mb0 + tid - 64].x;
            op_bar();  // rows and maxima of the block before are written, its tables read
            if (tid < b.nb0 + b.nb1) {
                tn[tid] = e;
            } else if (tid >= 64 && tid < 64 + b.mcount) {
                const int m = b.mb0 + tid - 64;
                // |Q_l| <= max |Q_{l-1}| + beta max |Q_{l-2}|
                auto mx = [&](int lv, int mm) {
                    const uint32_t h = s_mx[(lv % 3) * TC_LMAX + mm];
                    return __hiloint2double((int)h, h ? -1 : 0);
                };
                double bd = 1.0;
                if (l > 0) {
                    if (m == l) bd = mx(l - 1, m - 1);
                    else if (m == l - 1) bd = mx(l - 1, m);
                    else bd = fma(beta, mx(l - 2, m), mx(l - 1, m));
                }
                const int eb = (int)((uint32_t)__double2hiint(bd * 1.03) >> 20) & 0x7ff;
                tm[tid - 64] = make_double2(beta, __hiloint2double(0, max(eb - 1022, -1000)));
            } else if (tid >= 128 && b.mb0 == 0 && b.n0 == 0) {
                for (int k = tid - 128; k <= l + 1 && k < TC_LMAX; k += TC_OPT - 128) s_mx[(l % 3) * TC_LMAX + k] = 0u;
            }
            op_bar();
            const int nq = (b.mcount + 3) >> 2, nu = nq + ((b.ncount + 7) >> 3);
            const int at0 = (TC_DG * b.nb0 + 63) >> 6, natoms = at0 + ((TC_DG * b.nb1 + 63) >> 6);
            // written and read in this kernel: no read-only loads
            double *rw0 = a.rows + (size_t)(l & 1) * lset;  // Q_{l-2}, overwritten by Q_l
            const double *rw1 = a.rows + (size_t)((l + 1) & 1) * lset;
            const double2 *__restrict__ tab = LERP ? a.tab + (size_t)l * a.npts : nullptr;
            const bool first = b.n0 == 0;  // this block advances the rows; later n-blocks read them
            // The rows and phases of a warp's unit are loaded while the digits of its unit before are
            // stored: the L2's latency (~1000 cycles) is a third of a unit otherwise.
            double q[4], q2[4];
            ulonglong2 ph[4];
            auto load_next = [&](int t, int u) {  // this warp's unit after unit u of tile t (zeros if it is none of m)
                u += TC_OPW;
                while (u >= nu) {
                    u -= nu;
                    ++t;
                }
                const bool go = t < t1 && u < nq;
                const int m0 = b.mb0 + 4 * u;
                const uint32_t r0 = ((uint32_t)t * a.lmp + m0) * TC_KT + lane;
#pragma unroll
                for (int h = 0; h < 4; ++h) ph[h] = ld_if(a.phase + r0 + h * TC_KT, go);
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    // the first n-block reads Q_{l-1}, Q_{l-2}; later ones Q_l
                    q[h] = ld_if(first ? rw1 + r0 + (m0 + h == l ? h - 1 : h) * TC_KT : rw0 + r0 + h * TC_KT,
                                 go && m0 + h <= l && (l > 0 || !first));
                    q2[h] = ld_if(rw0 + r0 + h * TC_KT, go && first && m0 + h <= l - 2);
                }
                if (go && t + 2 < t1) {
                    // the same of the tile after next into L2: 32 lines, one per lane
                    const uint32_t rp = r0 - lane + 2u * a.lmp * TC_KT;
                    const char *pf = lane < 16   ? reinterpret_cast<const char *>(a.phase + rp) + lane * 128
                                     : lane < 24 ? reinterpret_cast<const char *>(rw1 + rp) + (lane - 16) * 128
                                                 : reinterpret_cast<const char *>(rw0 + rp) + (lane - 24) * 128;
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(pf));
                }
            };
            {
                int u = warp - ofs;
                if (u < 0) u += TC_OPW;
                load_next(t0, u - TC_OPW);
            }
            double2 xs = __ldg(a.xs + (size_t)t0 * TC_KT + lane);
            uint64_t r = __ldg(a.rint + (size_t)t0 * TC_KT + lane);
            for (int t = t0; t < t1; ++t) {
                const uint32_t bf = use & 1u, it = use >> 1;
                ++use;
                int u = warp - ofs;
                if (u < 0) u += TC_OPW;
                ofs = (ofs + nu) % TC_OPW;
                // every warp takes part in every tile, with or without a unit of it: none falls so far
                // behind that a barrier's parity would mean another phase.  The buffer is waited for
                // when a unit's digits are ready.
                bool mine = it == 0;
                const bool any = u < nu;
                uint8_t *sy = sm + bf * TC_BUF, *sj = sy + TC_SY;
                for (; u < nu; u += TC_OPW) {
                    uint64_t v[8];
                    if (u < nq) {
                        // four complex m at this point: rows 8 u .. 8 u + 7
                        const int m0 = b.mb0 + 4 * u;
                        if (first) {
                            const uint32_t r0 = ((uint32_t)t * a.lmp + m0) * TC_KT + lane;
                            uint32_t mh[4];
#pragma unroll
                            for (int h = 0; h < 4; ++h) {
                                q[h] = fma(m0 + h == l ? xs.y : xs.x, q[h], -tm[4 * u + h].x * q2[h]);
                                if (l == 0) q[h] = 1.0;
                                if (m0 + h <= l) rw0[r0 + h * TC_KT] = q[h];
                                mh[h] = __reduce_max_sync(0xffffffffu, (uint32_t)__double2hiint(q[h]) & 0x7fffffffu);
                            }
                            if (lane < 4 && m0 + lane <= l)
                                atomicMax(&s_mx[(l % 3) * TC_LMAX + m0 + lane],
                                          lane & 2 ? (lane & 1 ? mh[3] : mh[2]) : (lane & 1 ? mh[1] : mh[0]));
                        }
#pragma unroll
                        for (int h = 0; h < 4; ++h) {
                            // |q| 2^(61 - EP), then times the 58-bit phase, upper 64 bits: < 2^55
                            const uint32_t qh = (uint32_t)__double2hiint(q[h]), ql = (uint32_t)__double2loint(q[h]);
                            const int s = __double2loint(tm[4 * u + h].y) + 1022 - (int)((qh >> 20) & 0x7ffu);
                            const uint64_t mant = ((uint64_t)((qh & 0xfffffu) | 0x100000u) << 40) | ((uint64_t)ql << 8);
                            const uint64_t p = shr64(mant, s);
                            // both factors as signed halves: three products, no sign to carry along
                            const uint64_t ps = signed_halves(qh >> 31 ? -(int64_t)p : (int64_t)p);
                            const int32_t p1 = (int32_t)(ps >> 32), p0 = (int32_t)ps;
                            auto prod = [&](uint64_t c) {
                                const int32_t c1 = (int32_t)(c >> 32), c0 = (int32_t)c;
                                const int64_t t2 = (int64_t)p1 * c0 + ((int64_t)p0 * c1 + 0x80000000ll);  // rounded
                                return (uint64_t)((int64_t)p1 * c1 + ((t2 >> 32) + (int64_t)TC_OFF_Y));
                            };
                            v[2 * h] = prod(ph[h].x);
                            v[2 * h + 1] = prod(ph[h].y);
                        }
                    } else {
                        // eight radial orders at this point
                        const int o = u - nq;
                        if (LERP) {
#pragma unroll
                            for (int h0 = 0; h0 < 8; h0 += 4) {
                                double2 y[4];
                                double f[4];
#pragma unroll
                                for (int h = 0; h < 4; ++h) {
                                    const uint4 kd = tn[8 * o + h0 + h];
                                    y[h] = __ldg(tab + lerp_at(r, kd, a.npts, f[h]));
                                }
#pragma unroll
                                for (int h = 0; h < 4; ++h)
                                    v[h0 + h] = j_digits(fma(y[h].y, f[h], y[h].x), tn[8 * o + h0 + h].w);
                            }
                        } else {
                            const size_t row = ((size_t)(l - a.l0) * a.tiles + t) * a.nmax + b.n0 + 8 * o;
                            const uint64_t *jp = a.jarr + row * TC_KT + lane;
#pragma unroll
                            for (int h = 0; h < 8; ++h) v[h] = 8 * o + h < b.ncount ? __ldg(jp + h * TC_KT) : TC_OFF_J;
                        }
                    }
                    load_next(t, u);
                    if (!mine) wait(&empty[bf], (it - 1) & 1, dead);
                    mine = true;
                    if (u < nq) {
                        const uint32_t atom = (uint32_t)u >> 3, c = (uint32_t)u & 7u;
                        uint8_t *dst = sy + (lk * 2 + atom) * 1024u + lr * 128u + ((c ^ lr) << 4);
                        Digits<0, TC_DY>::each([&](int d) { return dst + d * TC_YD; }, v);
                    } else {
                        // digit d's columns of a half start at d nb: an octet lies in one atom of 64
                        const int n = 8 * (u - nq), nbh = n < TC_NH ? b.nb0 : b.nb1;
                        uint8_t *dst = sj + (lk * (uint32_t)natoms + (n < TC_NH ? 0u : (uint32_t)at0)) * 1024u + lr * 128u;
                        uint32_t col = (uint32_t)(n & (TC_NH - 1));
                        Digits<0, TC_DG>::each(
                            [&](int) {
                                uint8_t *q8 = dst + (col >> 6) * 1024u + ((((col & 63u) >> 3) ^ lr) << 4);
                                col += (uint32_t)nbh;
                                return q8;
                            },
                            v);
                    }
                }
                if (t + 1 < t1) {  // the next tile's points
                    xs = __ldg(a.xs + (size_t)(t + 1) * TC_KT + lane);
                    r = __ldg(a.rint + (size_t)(t + 1) * TC_KT + lane);
                }
                if (any) {
                    tc05::fence_proxy_async();
                    __syncwarp();
                } else if (!mine) {
                    wait(&empty[bf], (it - 1) & 1, dead);
                }
                if (lane == 0) tc_arrive(&full[bf]);
            }
        });
        if (dead && lane == 0) *a.err = CATANA_ERR_CUDA;
        op_bar();
        for (int k = tid; k < 3 * TC_LMAX; k += TC_OPT) a.maxq[(size_t)slab * 3 * TC_LMAX + k] = s_mx[k];
    } else if (warp < TC_FOLD0) {
        uint32_t use = 0, groups = 0;  // tiles taken, groups issued
        bool dead = false;
        if (a.stall) wait(&drain, 0, dead);
        tc_blocks(a, [&](const TcBlock &b, int) {
            const uint32_t at0 = (uint32_t)(TC_DG * b.nb0 + 63) >> 6, natoms = at0 + ((uint32_t)(TC_DG * b.nb1 + 63) >> 6);
            for (int g = t0; g < t1; g += TC_GROUP) {
                const int ge = min(t1, g + TC_GROUP);
                for (int t = g; t < ge; ++t) {
                    const uint32_t bf = use & 1u;
                    wait(&full[bf], (use >> 1) & 1, dead);
                    ++use;
                    const uint32_t ya = tc05::smem_u32(sm + bf * TC_BUF), jb = ya + TC_SY;
                    for (uint32_t h = 0; h < (alt ? 1u : 2u); ++h) {
                        const uint32_t reg = alt ? groups & 1u : h, rn = alt ? groups >> 1 : groups;
                        // the region's group before is folded
                        if (t == g && rn > 0) wait(&dfree[reg], (rn - 1) & 1, dead);
                        if (lane == 0 && !dead) {
                            tc05::fence_after();
                            const uint32_t nbh = (uint32_t)(h ? b.nb1 : b.nb0), dt = tmem + reg * TC_DREG;
                            uint64_t da0 = tc05::desc_sw128(ya, 1024, 2048);
                            uint64_t db = tc05::desc_sw128(jb + (h ? at0 * 1024u : 0u), 1024, natoms * 1024u);
                            if (nbh) {
#pragma unroll
                                for (int ks = 0; ks < 2; ++ks) {
                                    uint32_t idesc = tc05::idesc_f16_mn(128, 0) + ((TC_DG * nbh >> 3) << 17), dc = dt;
#pragma unroll
                                    for (int ad = 0; ad < TC_DY; ++ad) {
                                        tc05::mma_f16(dc, da0 + (uint64_t)(ad * (TC_YD >> 4) + ks * 256), db, idesc,
                                                      (t > g || ks > 0 || ad > 0) ? 1u : 0u);
                                        dc += nbh;
                                        idesc -= (nbh >> 3) << 17;
                                    }
                                    db += natoms * 128u;
                                }
                            }
                            if (t + 1 == ge) tc05::commit(&gdone[reg]);
                        }
                        __syncwarp();
                    }
                    if (lane == 0 && !dead) tc05::commit(&empty[bf]);
                    __syncwarp();
                }
                ++groups;
            }
        });
        // Whatever was issued lands before the block's memory goes, also where a role gave up (bounded by the
        // drain limit, not by the possibly shortened limit of the waits above).
        if (lane == 0) {
            tc05::commit(&drain);
            tc05::mbar_wait(&drain, 0, TC_WAIT_NS);
            if (dead) *a.err = CATANA_ERR_CUDA;
        }
        __syncwarp();
    } else {
        uint32_t groups = 0;  // groups folded
        bool dead = false;
        const int qd = warp & 3, row = qd * 32 + lane;
        const uint32_t lane_off = (uint32_t)(qd * 32) << 16;
        // Slab sums are kept in units of 2^64, 2^-54 of the largest term: a group adds at most 2^61, and what
        // passes 2^60 goes to a count per sum (signed bytes, four to a word; at most two a group).
        // relative to the call's largest, which k_ptc_reduce applies: 2^(EP + EW) leaves FP64's range otherwise
        const int ew = a.slab[slab].ew + 2048 - a.call->etop;
        const int set = warp >= TC_FOLD0 + 4 ? 1 : 0;
        tc_blocks(a, [&](const TcBlock &b, int seq) {
            const bool live = qd * 32 < 2 * b.mcount;  // warp-uniform: the quadrant holds rows of the block
            // this warp's radial orders of the block, and their column in the region
            const int nbh = !alt && set ? b.nb1 : b.nb0, ncol = alt ? nbh >> 1 : nbh, col0 = alt ? set * ncol : 0;
            const int nb = alt ? col0 : set * TC_NH;
            int64_t acc[TC_NH];
#pragma unroll
            for (int c = 0; c < TC_NH; ++c) acc[c] = 0;
            int top[TC_NH / 4];
#pragma unroll
            for (int c = 0; c < TC_NH / 4; ++c) top[c] = 0;
            for (int g = t0; g < t1; g += TC_GROUP) {
                const uint32_t reg = alt ? groups & 1u : (uint32_t)set, rn = alt ? groups >> 1 : groups;
                wait(&gdone[reg], rn & 1, dead);
                ++groups;
                if (!dead && live) {
                    tc05::fence_after();
                    const uint32_t dt = tmem + reg * TC_DREG + lane_off + (uint32_t)col0;
#pragma unroll
                    for (int c2 = 0; c2 < TC_NH; c2 += 2) {
                        if (c2 < ncol) {
                            uint32_t d[TC_DG][2];
#pragma unroll
                            for (int k = 0; k < TC_DG; ++k) tmem_ld2(dt + (uint32_t)(k * nbh + c2), d[k]);
                            tc05::tmem_wait_ld();
#pragma unroll
                            for (int k = 0; k < 2; ++k) {
                                int iv[TC_DG];
#pragma unroll
                                for (int ad = 0; ad < TC_DG; ++ad) iv[ad] = __float2int_rn(__uint_as_float(d[ad][k]));
                                // sum_d iv_d 2^(56 - 8 d) in units of 2^16, the lowest digits rounded off
                                const int low = iv[5] + ((iv[6] + ((iv[7] + 128) >> 8) + 128) >> 8);
                                int64_t v = low + (int64_t)iv[4] * 256;
                                v += (int64_t)iv[3] * 65536;
                                v += (int64_t)iv[2] * 16777216;
                                v += (int64_t)(iv[0] * 256 + iv[1]) << 32;
                                v += acc[c2 + k];
                                const int hi = ((int)(v >> 32) + (1 << 27)) >> 28;  // multiples of 2^60, to nearest
                                acc[c2 + k] = v - ((int64_t)hi << 60);
                                top[(c2 + k) >> 2] += hi << (8 * ((c2 + k) & 3));
                            }
                        }
                    }
                }
                tc05::fence_before();
                tc_arrive(&dfree[reg]);
            }
            // the slab's sums: value = (acc + top 2^60) 2^(-54 + EJ + EP + EW) A_lm
            if (live && row < 2 * b.mcount) {
                const int ring = seq & (int)(TC_RING - 1);
                const uint4 *tn = s_n + ring * TC_NB + nb;
                const int m = b.mb0 + (row >> 1);
                const double am = scalbn(a.coef[(size_t)b.l * (b.l + 1) / 2 + m].y,
                                         __double2loint(s_m[ring * TC_MB + (row >> 1)].y) + ew);
                const int w2 = 2 * (b.l + 1);
                double *out = a.partial + (size_t)slab * a.pslab +
                              (size_t)a.nmax * ((size_t)b.l * (b.l + 1) - (size_t)a.l0 * (a.l0 + 1)) + 2 * b.mb0 + row +
                              (size_t)(b.n0 + nb) * w2;
#pragma unroll
                for (int c4 = 0; c4 < TC_NH; c4 += 4)
                    if (c4 < ncol) {
                        double v[4];
#pragma unroll
                        for (int c = 0; c < 4; ++c) v[c] = (double)acc[c4 + c];
                        if (__any_sync(__activemask(), top[c4 >> 2] != 0)) {
                            int x = top[c4 >> 2];
#pragma unroll
                            for (int c = 0; c < 4; ++c) {
                                const int y = (int)(int8_t)x;
                                v[c] = fma((double)y, 0x1p60, v[c]);
                                x = (x - y) >> 8;
                            }
                        }
#pragma unroll
                        for (int c = 0; c < 4; ++c)  // 2^(EJ - 54) is a normal number: EJ >= -900
                            v[c] *= __hiloint2double((int)(tn[c4 + c].w - (53u << 20)), 0);
#pragma unroll
                        for (int c = 0; c < 4; ++c)
                            if (nb + c4 + c < b.ncount) out[(size_t)(c4 + c) * w2] = v[c] * am;
                    }
            }
        });
        if (dead && lane == 0) *a.err = CATANA_ERR_CUDA;
    }
    tc05::fence_before();
    __syncthreads();
    tc05::fence_after();
    if (warp == TC_FOLD0) tc05::tmem_dealloc(tmem, tcols);
}

// Per (slab, l, n): the table's step (k / dx as 62-bit mantissa and shift) and the exponent bound of
// |j_l(k r)| over the slab's radii.  With the table, a slab that reaches past it is a domain error.
__global__ void __launch_bounds__(128) k_ptc_ntab(const TcSlab *__restrict__ slab, const double *__restrict__ kln,
                                                  const double *__restrict__ dxinv, const double *__restrict__ zmax, int l0,
                                                  int nl, int nmax, int er, uint4 *__restrict__ out, int *err) {
    const int e = blockIdx.y * 128 + threadIdx.x;
    if (e >= nl * nmax) return;
    const int l = l0 + e / nmax, n = e % nmax;
    const TcSlab sl = slab[blockIdx.x];
    const double k = kln[(size_t)l * nmax + n];
    float z1 = (float)(k * sl.rmin), z2 = (float)(k * sl.rmax);
    uint4 o = make_uint4(0u, 0u, 31u, 0u);
    if (dxinv) {
        const double kd = k * dxinv[l];
        const float dx = 1.f / (float)dxinv[l];
        z1 = fmaxf(z1 - 1.0001f * dx, 0.f);  // interpolated values lie between nodes up to dx away
        z2 += 1.0001f * dx;
        const uint64_t bits = (uint64_t)__double_as_longlong(kd);
        const int ek = (int)(bits >> 52) - 1022;  // kd in [2^(ek - 1), 2^ek)
        const uint64_t kdi = ((bits & 0xfffffffffffffull) | 0x10000000000000ull) << 9;  // kd 2^(62 - ek)
        o.x = (uint32_t)(kdi >> 32);
        o.y = (uint32_t)kdi;
        o.z = (uint32_t)(4 + er + ek);  // k r / dx = (rint kdi / 2^64) / 2^(60 - er - ek)
        if (n == nmax - 1 && k * sl.rmax >= zmax[l]) *err = CATANA_ERR_DOMAIN;
    }
    const float lb = jl_log2_bound(l, z1, z2 * 1.000001f) + 0.03f;
    o.w = (uint32_t)(max(-900, (int)floorf(lb) + 1 + sl.ec) + 1022) << 20;
    out[(size_t)blockIdx.x * nl * nmax + e] = o;
}

// Sort keys: r / rmax on 2^bits steps (radii past rmax share the last one).
__global__ void k_ptc_keys(const double *__restrict__ pts, int64_t n, double inv_rmax, int bits,
                           uint32_t *keys, uint32_t *vals) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double top = (double)(1 << bits);
    const double q = fabs(pts[3 * i]) * inv_rmax * top;
    keys[i] = q >= top - 1.0 ? (1u << bits) - 1u : (q > 0.0 ? (uint32_t)q : 0u);
    vals[i] = (uint32_t)i;
}

// Per slab: range of |r| and exponent of the largest |w|.  Values that are not finite are left out (they
// poison the result, k_ptc_points); so are, with the table, radii outside it (a domain error).
__global__ void __launch_bounds__(256) k_ptc_slabs(const double *__restrict__ pts, const double *__restrict__ w,
                                                   const uint32_t *__restrict__ perm, int64_t n, int64_t per, double rlim,
                                                   TcSlab *__restrict__ out, TcCall *__restrict__ call) {
    const int64_t i0 = blockIdx.x * per, i1 = min(n, i0 + per);
    double lo = INFINITY, hi = 0.0, mw = 0.0;
    for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
        const int64_t j = perm[i];
        const double r = fabs(pts[3 * j]);
        if (r < rlim) {  // false for NaN
            lo = fmin(lo, r);
            hi = fmax(hi, r);
        }
        const double v = w ? fabs(w[j]) : 1.0;
        if (isfinite(v)) mw = fmax(mw, v);
    }
    __shared__ double s[3][8];
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        mw = fmax(mw, __shfl_xor_sync(0xffffffffu, mw, o));
    }
    if ((threadIdx.x & 31) == 0) {
        s[0][threadIdx.x >> 5] = lo;
        s[1][threadIdx.x >> 5] = hi;
        s[2][threadIdx.x >> 5] = mw;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) {
            lo = fmin(lo, s[0][k]);
            hi = fmax(hi, s[1][k]);
            mw = fmax(mw, s[2][k]);
        }
        TcSlab o;
        o.rmin = lo <= hi ? lo : 0.0;
        o.rmax = hi;
        o.ew = mw > 0.0 ? ilogb(mw) + 1 : -1100;  // mw < 2^ew
        o.ec = 0;
        atomicMax(&call->etop, 2048 + o.ew);
        out[blockIdx.x] = o;
    }
}

// A catalog in RING pixels (k_ptc_pixels).  Its points share their pixels' centres, so what the main kernel
// takes as a point is an entry: up to TC_CELL points of one pixel, whose j_l are summed first (k_ptc_jl_cells).
constexpr int TC_CELL = 64;
struct TcPixels {
    const double *r;            // radii grouped by pixel
    const int64_t *offs;        // [npix + 1]
    int64_t npix;
    int nrings, lmax, conj;
    const int64_t *ring_start;  // first pixel
    const int *ring_pix;        // pixels
    const double *ring_x;       // cos theta
    const double2 *ring_ph;     // [m][ring]: e^{-i m phi_0}
    const double2 *tw;          // e^{-2 pi i k / N} per ring length, at tw_off[ring]
    const int64_t *tw_off;
};

constexpr int TC_POISON_THETA = 1, TC_POISON_PHI = 2, TC_POISON_W = 4;

// v = w 2^-ew cos or -w 2^-ew sin of m phi, times 2^58, in signed halves
__device__ __forceinline__ uint64_t phase_word(double v) { return signed_halves(__double2ll_rn(v * 0x1p58)); }

// Point records and phase tables, in sorted order: a warp per (tile, run of 8 m), lane = point.  The
// phase of the run's middle comes from the exactly reduced fraction frac(m phi / 2 pi) and is rotated
// by e^{+-i phi} for the others (at most four times).
__global__ void __launch_bounds__(256) k_ptc_points(const double *__restrict__ pts, const double *__restrict__ w,
                                                    const uint32_t *__restrict__ perm, int64_t n, int tiles, int tslab,
                                                    int lmp, const TcSlab *__restrict__ slab, int er, int lerp,
                                                    double rlim, uint64_t *__restrict__ rint, double *__restrict__ rabs,
                                                    double2 *__restrict__ xs, ulonglong2 *__restrict__ phase,
                                                    TcCall *__restrict__ call, int *__restrict__ err) {
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= tiles) return;
    const int64_t i = (int64_t)t * TC_KT + lane;
    const bool in = i < n;
    const int64_t j = in ? perm[i] : perm[n - 1];  // padding takes the last point's radius and no weight
    const double r = pts[3 * j], th = pts[3 * j + 1], ph = pts[3 * j + 2];
    double wv = in ? (w ? w[j] : 1.0) : 0.0;
    int bad = 0;
    if (!isfinite(th)) bad |= TC_POISON_THETA;
    if (!isfinite(ph)) bad |= TC_POISON_PHI;
    if (!isfinite(wv)) bad |= TC_POISON_W;
    const bool rbad = lerp ? !(r >= 0.0 && r < rlim) : !isfinite(r);
    if (rbad && !lerp) bad |= TC_POISON_W;
    // An angle that is not finite spoils the modes that it enters (k_ptc_reduce makes them NaN); the others, l = 0
    // for theta and m = 0 for phi, keep the point.
    const bool use = in && !(bad & TC_POISON_W) && !rbad;
    const double ct = cos(th);
    if (blockIdx.y == 0) {
        if (in && bad) atomicOr(&call->poison, bad);
        if (in && rbad && lerp) *err = CATANA_ERR_DOMAIN;  // outside every table
        rint[i] = rbad || !(fabs(r) < ldexp(1.0, er)) ? 0ull : (uint64_t)(int64_t)ldexp(fmax(r, 0.0), 62 - er);
        rabs[i] = r;
        xs[i] = use && !(bad & TC_POISON_THETA) ? make_double2(ct, sqrt((1.0 - ct) * (1.0 + ct))) : make_double2(0.0, 0.0);
    }
    const int e = -slab[t / tslab].ew;
    wv = use ? wv * pow2_lo(e) * pow2_hi(e) : 0.0;  // in [-1, 1], exact for weights of any size
    const double phi = use && !(bad & TC_POISON_PHI) ? ph : 0.0;
    // frac(phi / 2 pi) 2^64 (mod 2^64), 1 / 2 pi as a pair of doubles: rounded at 2^-64 of a turn
    const double p = phi * 0.15915494309189535, pl = fma(phi, 0.15915494309189535, -p) - phi * 9.839338337591243e-18;
    const double f = p - floor(p);
    const unsigned long long u = (f < 1.0 ? (unsigned long long)ldexp(f, 64) : 0ull) +
                                 (unsigned long long)__double2ll_rn(fabs(pl) < 0.25 ? ldexp(pl, 64) : 0.0);
    double s1, c1;
    sincos(phi, &s1, &c1);
    const int m0 = blockIdx.y * 8, mc = m0 + 4;
    double sn, cs;
    sincospi((double)(long long)((unsigned long long)mc * u) * 1.0842021724855044340074528008699e-19, &sn, &cs);  // 2^-63
    ulonglong2 *o = phase + ((size_t)t * lmp + m0) * TC_KT + lane;
    double er_ = cs * wv, ei = -sn * wv;
    double ur = er_, ui = ei;
    for (int k = 4; k < 8 && m0 + k < lmp; ++k) {
        o[k * TC_KT] = make_ulonglong2(phase_word(ur), phase_word(ui));
        const double nr = ur * c1 + ui * s1, ni = ui * c1 - ur * s1;
        ur = nr;
        ui = ni;
    }
    for (int k = 3; k >= 0; --k) {
        const double nr = er_ * c1 - ei * s1, ni = ei * c1 + er_ * s1;
        er_ = nr;
        ei = ni;
        if (m0 + k < lmp) o[k * TC_KT] = make_ulonglong2(phase_word(er_), phase_word(ei));
    }
}

// last pixel with offs[p] <= q
__device__ __forceinline__ int64_t pixel_of(const TcPixels &px, int64_t q) {
    int64_t lo = 0, hi = px.npix;
    while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (px.offs[mid] <= q) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Sort keys of a pixelized catalog: every TC_CELL-th point of a pixel heads an entry, the fullest entries
// first (a warp sums as long as its longest), of like ones by the head's radius in 256 steps (the lanes of a
// warp then share cells of the j_l table where entries hold few points: 34 -> 32 ms below); the other points
// come last.  Also each radius in the table's units.
__global__ void k_ptc_cells(TcPixels px, int64_t n, double inv_rmax, int er, int lerp, double rlim,
                            uint32_t *__restrict__ keys, uint32_t *__restrict__ vals, uint64_t *__restrict__ rint,
                            TcCall *__restrict__ call, int *__restrict__ err) {
    const int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int64_t p = q < n ? pixel_of(px, q) : 0, k = q < n ? q - px.offs[p] : 1;
    // every thread of the block takes part, whatever its bisection took
    const int heads = __syncthreads_count(k % TC_CELL == 0);
    if (threadIdx.x == 0 && heads) atomicAdd(&call->count, (unsigned long long)heads);
    if (q >= n) return;
    const double r = px.r[q], rs = r * inv_rmax * 256.0;
    const uint32_t rb = rs >= 255.0 ? 255u : (rs > 0.0 ? (uint32_t)rs : 0u);
    const int64_t cnt = k % TC_CELL == 0 ? min((int64_t)TC_CELL, px.offs[p + 1] - q) : 0;
    keys[q] = (uint32_t)(TC_CELL - cnt) << 8 | rb;
    vals[q] = (uint32_t)q;
    const bool bad = lerp ? !(r >= 0.0 && r < rlim) : !isfinite(r);
    if (bad && lerp) *err = CATANA_ERR_DOMAIN;  // outside every table
    if (bad && !lerp) atomicOr(&call->poison, TC_POISON_W);
    rint[q] = bad || !(fabs(r) < ldexp(1.0, er)) ? 0ull : (uint64_t)(int64_t)ldexp(fmax(r, 0.0), 62 - er);
}

// Per slab of entries what k_ptc_slabs finds for points (weights are 1)
__global__ void __launch_bounds__(256) k_ptc_cell_slabs(TcPixels px, const uint2 *__restrict__ cell, int64_t n, int64_t per,
                                                        double rlim, TcSlab *__restrict__ out,
                                                        TcCall *__restrict__ call) {
    const int64_t i0 = blockIdx.x * per, i1 = min(n, i0 + per);
    double lo = INFINITY, hi = 0.0;
    for (int64_t i = i0 + threadIdx.x; i < i1; i += blockDim.x) {
        const uint2 c = cell[i];
        for (uint32_t k = 0; k < c.y; ++k) {
            const double r = fabs(px.r[(int64_t)c.x + k]);
            if (r < rlim) {  // false for NaN
                lo = fmin(lo, r);
                hi = fmax(hi, r);
            }
        }
    }
    __shared__ double s[2][8];
    for (int o = 16; o > 0; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        s[0][threadIdx.x >> 5] = lo;
        s[1][threadIdx.x >> 5] = hi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k) {
            lo = fmin(lo, s[0][k]);
            hi = fmax(hi, s[1][k]);
        }
        TcSlab o;
        o.rmin = lo <= hi ? lo : 0.0;
        o.rmax = hi;
        o.ew = 1;
        atomicMax(&call->etop, 2048 + o.ew);
        o.ec = 32 - __clz((int)cell[i0].y - 1);  // the slab's first entry is its fullest
        out[blockIdx.x] = o;
    }
}

// The same as k_ptc_points for the entries of a catalog in RING pixels, at their pixels' centres: (ring's cos
// theta, phase e^{-i m phi_0} e^{-2 pi i j s / N}) with phi_0 the ring's first centre, j the pixel's place among
// the ring's N and s the frequency that the m-extraction reads (sfb_reverse_fft.cpp:192-207): m mod N up to
// N / 2, then N - m mod N, conjugated only where `conj` says so.  Both factors come from tables (ring_ph, tw).
__global__ void __launch_bounds__(256) k_ptc_pixels(TcPixels px, const uint32_t *__restrict__ perm, int64_t n,
                                                    int tiles, int lmp, uint2 *__restrict__ cell, double2 *__restrict__ xs,
                                                    ulonglong2 *__restrict__ phase) {
    const int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= tiles) return;
    const int64_t i = (int64_t)t * TC_KT + lane;
    const bool use = i < n;
    const int64_t q = use ? perm[i] : perm[n - 1];
    const int64_t lo = pixel_of(px, q);
    int ra = 0, rb = px.nrings;
    while (rb - ra > 1) {
        const int mid = (ra + rb) >> 1;
        if (px.ring_start[mid] <= lo) ra = mid;
        else rb = mid;
    }
    if (blockIdx.y == 0) {
        const double x = px.ring_x[ra];
        cell[i] = make_uint2((uint32_t)q, use ? (uint32_t)min((int64_t)TC_CELL, px.offs[lo + 1] - q) : 0u);
        xs[i] = use ? make_double2(x, sqrt((1.0 - x) * (1.0 + x))) : make_double2(0.0, 0.0);
    }
    const double w = use ? 0.5 : 0.0;  // unit weights: ew = 1
    const int N = px.ring_pix[ra], j = (int)(lo - px.ring_start[ra]);
    const double2 *tw = px.tw + px.tw_off[ra];
    const int m0 = blockIdx.y * 8;
    ulonglong2 *o = phase + ((size_t)t * lmp + m0) * TC_KT + lane;
    for (int k = 0; k < 8 && m0 + k < lmp; ++k) {
        const int m = m0 + k, mm = m % N, s = 2 * mm > N ? N - mm : mm;
        double2 a = make_double2(0.0, 0.0), f = a;
        if (m < px.lmax) {
            a = px.ring_ph[(size_t)m * px.nrings + ra];
            f = tw[(int)((int64_t)j * s % N)];
            if (px.conj && 2 * mm > N) f.y = -f.y;
        }
        o[k * TC_KT] = make_ulonglong2(phase_word(w * (a.x * f.x - a.y * f.y)), phase_word(w * (a.x * f.y + a.y * f.x)));
    }
}

// e^{-i m phi_0} per (m, ring)
__global__ void k_ptc_ring_phases(const double *__restrict__ ring_phi, int nrings, int lmax, double2 *__restrict__ o) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nrings * lmax) return;
    const int m = t / nrings;
    double sn, cs;
    sincos((double)m * ring_phi[t - m * nrings], &sn, &cs);
    o[t] = make_double2(cs, -sn);
}

// (y0 - dy, dy) per node of the linear tables; the last node is empty
__global__ void k_ptc_pairs(const double *__restrict__ y, int npts, int64_t total, double2 *__restrict__ o) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= total) return;
    if ((int)(t % npts) == npts - 1) {
        o[t] = make_double2(0.0, 0.0);
        return;
    }
    const double d = y[t + 1] - y[t];
    o[t] = make_double2(y[t] - d, d);
}

// f[l][m][n] += k_ln sum over slabs, in eight interleaved parts added in order; one CTA per 32 (m, n) of
// a level.  Points that are not finite make their terms NaN: theta every l > 0, phi every m > 0, w all.
__global__ void __launch_bounds__(256) k_ptc_reduce(const double *__restrict__ partial, int64_t pslab, int nslabs, int l0,
                                                    int nmax, const double *__restrict__ kln, const TcCall *__restrict__ call,
                                                    double2 *__restrict__ f) {
    __shared__ double2 s[8][33];
    const int l = l0 + blockIdx.y, cnt = (l + 1) * nmax;
    const int64_t base = (int64_t)nmax * ((int64_t)l * (l + 1) - (int64_t)l0 * (l0 + 1));
    const int lane = threadIdx.x & 31, part = threadIdx.x >> 5;
    for (int e0 = blockIdx.x * 32; e0 < cnt; e0 += gridDim.x * 32) {
        const int e = e0 + lane;  // n (l + 1) + m
        double sr = 0.0, si = 0.0;
        if (e < cnt) {
            const double2 *p = reinterpret_cast<const double2 *>(partial + base) + e;
#pragma unroll 4
            for (int k = part; k < nslabs; k += 8) {
                const double2 v = p[(size_t)k * (pslab / 2)];
                sr += v.x;
                si += v.y;
            }
        }
        s[part][lane] = make_double2(sr, si);
        __syncthreads();
        if (part == 0 && e < cnt) {
#pragma unroll
            for (int k = 1; k < 8; ++k) {
                sr += s[k][lane].x;
                si += s[k][lane].y;
            }
            const int n = e / (l + 1), m = e - n * (l + 1);
            const double k = kln[(size_t)l * nmax + n];
            double2 *o = f + (size_t)nmax * l * (l + 1) / 2 + (size_t)m * nmax + n;
            const int bad = call->poison, e = call->etop - 2048;
            double2 v = *o;
            if ((bad & TC_POISON_W) || ((bad & TC_POISON_THETA) && l > 0) || ((bad & TC_POISON_PHI) && m > 0)) {
                v = make_double2(NAN, NAN);
            } else {
                const double ks = k * pow2_lo(e);
                v.x += ks * sr * pow2_hi(e);
                v.y += ks * si * pow2_hi(e);
            }
            *o = v;
        }
        __syncthreads();
    }
}

// J of every (l, n, point) of the launch's levels: a warp per (l, tile, n), lane = point
struct TcJ {
    const double *r, *kln;
    const uint64_t *rint;
    const uint4 *ntab;
    int l0, nl, nmax, tiles, tslab, er;
    uint64_t *out;
    const uint2 *cell;   // pixelized catalogs: (first point, points) of each entry
    const double2 *tab;  // and the linear tables [l][npts], or null
    int npts;
};
__device__ __forceinline__ bool tc_j_index(const TcJ &a, int &l, int &t, int &n, size_t &e) {
    const int64_t q = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (q >= (int64_t)a.nl * a.tiles * a.nmax) return false;  // warp-uniform
    n = (int)(q % a.nmax);
    const int64_t q2 = q / a.nmax;
    t = (int)(q2 % a.tiles);
    l = a.l0 + (int)(q2 / a.tiles);
    e = (size_t)q * TC_KT + (threadIdx.x & 31);
    return true;
}
__global__ void __launch_bounds__(256) k_ptc_jl_exact(TcJ a) {
    int l, t, n;
    size_t e;
    if (!tc_j_index(a, l, t, n, e)) return;
    const double z = a.kln[(size_t)l * a.nmax + n] * a.r[(size_t)t * TC_KT + (threadIdx.x & 31)];
    const uint32_t w = a.ntab[((size_t)(t / a.tslab) * a.nl + (l - a.l0)) * a.nmax + n].w;
    a.out[e] = j_digits(isfinite(z) ? jl_direct(l, z) : 0.0, w);
}

// J of a pixelized catalog's entries, the sums over their points, exact in units of 2^-63 of the bound (which
// leaves room for the count).  With the tables a warp takes four radial orders of a tile (with eight, or two, the
// registers and the radii read again cost as much: 114.3 and 120.4 ms a call against 113.4).  What bounds it are
// the table's gathers from L2, most of them of unsorted radii, and ~60 instructions a value.  1M points on nside
// 256, l 128, n 64: 31 ms, and the main kernel over 0.57M entries 78 ms; over 1M points with their j_l 165.
constexpr int JC_N = 4;
__global__ void __launch_bounds__(256, 4) k_ptc_jl_cells(TcJ a) {
    const int lane = threadIdx.x & 31, noct = (a.nmax + JC_N - 1) / JC_N;
    const int64_t q = blockIdx.x * (int64_t)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (q >= (int64_t)a.nl * a.tiles * noct) return;  // warp-uniform
    const int o = (int)(q % noct);
    const int64_t q2 = q / noct;
    const int t = (int)(q2 % a.tiles), lv = (int)(q2 / a.tiles), nc = min(JC_N, a.nmax - JC_N * o);
    const uint4 *kp = a.ntab + ((size_t)(t / a.tslab) * a.nl + lv) * a.nmax + JC_N * o;
    const double2 *__restrict__ tab = a.tab + (size_t)(a.l0 + lv) * a.npts;
    const uint2 c = a.cell[(size_t)t * TC_KT + lane];
    uint64_t v[JC_N];
    uint4 kd[JC_N];
#pragma unroll
    for (int h = 0; h < JC_N; ++h) {
        v[h] = TC_OFF_J;
        kd[h] = __ldg(kp + min(h, nc - 1));
    }
    for (uint32_t k = 0; k < c.y; ++k) {
        const uint64_t r = __ldg(a.rint + (size_t)c.x + k);
        double2 y[JC_N];
        double f[JC_N];
#pragma unroll
        for (int h = 0; h < JC_N; ++h) y[h] = __ldg(tab + lerp_at(r, kd[h], a.npts, f[h]));
#pragma unroll
        for (int h = 0; h < JC_N; ++h) v[h] += j_digits(fma(y[h].y, f[h], y[h].x), kd[h].w) - TC_OFF_J;
    }
    uint64_t *out = a.out + (((size_t)lv * a.tiles + t) * a.nmax + JC_N * o) * TC_KT + lane;
#pragma unroll
    for (int h = 0; h < JC_N; ++h)
        if (h < nc) out[h * TC_KT] = v[h];
}
__global__ void __launch_bounds__(256) k_ptc_jl_cells_exact(TcJ a) {
    int l, t, n;
    size_t e;
    if (!tc_j_index(a, l, t, n, e)) return;
    const uint32_t w = a.ntab[((size_t)(t / a.tslab) * a.nl + (l - a.l0)) * a.nmax + n].w;
    const double kl = a.kln[(size_t)l * a.nmax + n];
    const uint2 c = a.cell[(size_t)t * TC_KT + (threadIdx.x & 31)];
    uint64_t v = TC_OFF_J;
    for (uint32_t k = 0; k < c.y; ++k) {
        const double z = kl * a.r[(size_t)c.x + k];
        v += j_digits(isfinite(z) ? jl_direct(l, z) : 0.0, w) - TC_OFF_J;
    }
    a.out[e] = v;
}

// The FP64 polynomials (sfb_fp64.cu, sum_s a_s t^s on unit intervals, t in [-1, 1]) as integers: Horner's
// steps are 64-bit integer products here (~10 instructions each; an FP64 FMA occupies its pipe for 16
// cycles per warp).  With B_s = 4^s A_s K the step B_s = 4^s a_s K + t B_{s+1} / 4 is the upper half of
// t 2^62 times B_{s+1}; K = 2^(59 - e), max_s |4^s a_s| < 2^e, keeps |B_s| < 2^60.  The terms s >= 9 (below
// 1e-8 of the first) take 32-bit products at a scale of their own, and are shifted to the others' (up).
struct TcPoly {
    int64_t c[9];
    int32_t h[3];
    int32_t e, up, pad;
};
static_assert(sizeof(TcPoly) == 96, "TcPoly layout");

__global__ void k_ptc_poly_int(const double *__restrict__ poly, int64_t total, TcPoly *__restrict__ out) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= total) return;
    double a[12], mx = 0.0;
    for (int k = 0; k < 12; ++k) {
        a[k] = ldexp(poly[t * 12 + k], 2 * k);
        mx = fmax(mx, fabs(a[k]));
    }
    TcPoly o;
    o.e = mx > 0.0 ? ilogb(mx) + 1 : -2000;
    for (int k = 0; k < 9; ++k) o.c[k] = __double2ll_rn(ldexp(a[k], 59 - o.e));
    double mh = 0.0;
    for (int k = 9; k < 12; ++k) mh = fmax(mh, fabs(a[k]));
    const int e9 = mh > 0.0 ? ilogb(mh) + 1 : -2000;  // |4^s a_s| < 2^e9
    for (int k = 9; k < 12; ++k) o.h[k - 9] = __double2int_rn(ldexp(a[k], 29 - e9));
    o.up = 30 - o.e + e9;
    o.pad = 0;
    out[t] = o;
}

__global__ void __launch_bounds__(256) k_ptc_jl_poly(TcJ a, const TcPoly *__restrict__ poly, int nint, int *err) {
    int l, t, n;
    size_t e;
    if (!tc_j_index(a, l, t, n, e)) return;
    const uint64_t kb = (uint64_t)__double_as_longlong(a.kln[(size_t)l * a.nmax + n]);
    const uint64_t r = a.rint[(size_t)t * TC_KT + (threadIdx.x & 31)];
    const uint32_t w = a.ntab[((size_t)(t / a.tslab) * a.nl + (l - a.l0)) * a.nmax + n].w;
    // z = k r = (r kmant / 2^64) / 2^(60 - er - ek): integer and 64-bit fraction of z + 1/2
    const int sh = 4 + a.er + (int)(kb >> 52) - 1022;
    const uint64_t km = ((kb & 0xfffffffffffffull) | 0x10000000000000ull) << 9;
    const uint32_t kh = (uint32_t)(km >> 32), kl = (uint32_t)km, rh = (uint32_t)(r >> 32), rl = (uint32_t)r;
    const uint64_t tt = (uint64_t)rl * kh + (uint64_t)rh * kl, res = (uint64_t)rh * kh + (tt >> 32);
    // 60 - er - ek bits of res are fraction (up to 64: k r < 1/16 when sh < 0)
    const uint64_t low = (uint64_t)(uint32_t)tt << 32;
    uint64_t fr = sh >= 0 ? (res << sh) | (low >> (64 - sh) & (sh ? ~0ull : 0ull)) : shr64(res, -sh);
    uint32_t j = sh > 0 ? (uint32_t)(res >> (64 - sh)) : 0u;
    fr += 0x8000000000000000ull;
    j += fr < 0x8000000000000000ull ? 1u : 0u;
    if (j >= (uint32_t)nint) {  // the host sized the table from max r
        *err = CATANA_ERR_DOMAIN;
        j = 0;
    }
    const uint64_t ts = signed_halves((int64_t)(fr - 0x8000000000000000ull) >> 1);  // t 2^62
    const int32_t t1 = (int32_t)(ts >> 32), t0 = (int32_t)ts;
    const int4 *q = reinterpret_cast<const int4 *>(poly + (size_t)l * nint + j);
    const longlong2 c8 = __ldg(reinterpret_cast<const longlong2 *>(q + 4));  // c_8; h_9, h_10
    const int4 he = __ldg(q + 5);                                              // h_11, e, up
    int32_t b = he.x;
    b = (int32_t)(c8.y >> 32) + __mulhi(b, t1);
    b = (int32_t)c8.y + __mulhi(b, t1);
    int64_t v = he.z >= 0 ? (int64_t)b << min(he.z, 32) : (int64_t)(b >> min(-he.z, 31));
    auto step = [&](int64_t ck) {
        const uint64_t h = signed_halves(v);
        const int32_t h1 = (int32_t)(h >> 32), h0 = (int32_t)h;
        const int64_t m = (int64_t)h1 * t0 + ((int64_t)h0 * t1 + 0x80000000ll);
        v = (int64_t)h1 * t1 + ((m >> 32) + ck);
    };
    step(c8.x);
#pragma unroll
    for (int k = 3; k >= 0; --k) {
        const longlong2 c = __ldg(reinterpret_cast<const longlong2 *>(q + k));
        step(c.y);
        step(c.x);
    }
    // j_l = v 2^(e - 59) -> 2^(63 - EJ) j_l
    const int up = 4 + he.y - ((int)(w >> 20) - 1022);
    v = up >= 0 ? (up > 63 ? 0 : v << up) : v >> min(63, -up);
    a.out[e] = TC_OFF_J + (uint64_t)v;
}

size_t tc_al(size_t b) { return (b + 255) & ~size_t(255); }

// (beta, A) per (l, m): Q_l = x Q_{l-1} - beta Q_{l-2}, P = A Q, Q_mm = sin^m
catana_status_t ensure_tc_coefs(DeviceContext *ctx, int lmax, cudaStream_t st) {
    if (ctx->tc_coef_lmax >= lmax) return CATANA_OK;
    std::vector<double2> h((size_t)lmax * (lmax + 1) / 2);
    long double amm = 0.28209479177387814347403972578038630L;  // 1 / sqrt(4 pi)
    for (int m = 0; m < lmax; ++m) {
        if (m > 0) amm *= -sqrtl((2.0L * m + 1.0L) / (2.0L * m));
        long double A = amm;
        for (int l = m; l < lmax; ++l) {
            double beta = 0.0;
            if (l > m) {
                const long double dl = l, mm = (long double)m * m;
                A *= sqrtl((4.0L * dl * dl - 1.0L) / (dl * dl - mm));
            }
            if (l > m + 1) {
                const double d1 = l - 1;
                beta = (d1 * d1 - (double)m * m) / (4.0 * d1 * d1 - 1.0);
            }
            h[(size_t)l * (l + 1) / 2 + m] = make_double2(beta, (double)A);
        }
    }
    ctx->tc_coef_lmax = -1;
    CG_CUDA_TRY(ctx->tc_coef.ensure(h.size() * sizeof(double2)));
    CG_CUDA_TRY(cudaMemcpyAsync(ctx->tc_coef.ptr, h.data(), h.size() * sizeof(double2), cudaMemcpyHostToDevice, st));
    CG_CUDA_TRY(cudaStreamSynchronize(st));
    ctx->tc_coef_lmax = lmax;
    return CATANA_OK;
}

// (y0 - dy, dy) tables, dx^-1 and z_max per l (cached like the tables that they are made from)
catana_status_t ensure_tc_tables(DeviceContext *ctx, int lmax, int nmax, cudaStream_t st) {
    catana_status_t s = ensure_lerp_tables(ctx, lmax, nmax, st);
    if (s != CATANA_OK) return s;
    if (ctx->tc_tab_lmax >= lmax && ctx->tc_tab_nmax == nmax) return CATANA_OK;
    lmax = ctx->tab_lmax;
    const int npts = 1000 * nmax;
    const int64_t total = (int64_t)lmax * npts;
    const size_t tb = tc_al((size_t)total * sizeof(double2));
    ctx->tc_tab_lmax = ctx->tc_tab_nmax = -1;
    CG_CUDA_TRY(ctx->tc_tab.ensure(tb + 2 * (size_t)lmax * sizeof(double)));
    double *dz = reinterpret_cast<double *>(ctx->tc_tab.as<char>() + tb);
    k_ptc_pairs<<<ceil_div(total, 256), 256, 0, st>>>(ctx->tables.as<double>(), npts, total, ctx->tc_tab.as<double2>());
    count_launch();
    CG_CUDA_TRY(cudaGetLastError());
    CG_CUDA_TRY(cudaMemcpyAsync(dz, ctx->tab_dxinv.data(), lmax * sizeof(double), cudaMemcpyHostToDevice, st));
    CG_CUDA_TRY(cudaMemcpyAsync(dz + lmax, ctx->tab_zmax.data(), lmax * sizeof(double), cudaMemcpyHostToDevice, st));
    CG_CUDA_TRY(cudaStreamSynchronize(st));
    ctx->tc_tab_off = tb;
    ctx->tc_tab_lmax = lmax;
    ctx->tc_tab_nmax = nmax;
    return CATANA_OK;
}

// the polynomials of ctx->poly as integers (rebuilt when those are)
catana_status_t ensure_tc_poly(DeviceContext *ctx, cudaStream_t st) {
    if (ctx->tc_poly_lmax == ctx->poly_lmax && ctx->tc_poly_nint == ctx->poly_nint) return CATANA_OK;
    const int64_t total = (int64_t)ctx->poly_lmax * ctx->poly_nint;
    ctx->tc_poly_lmax = ctx->tc_poly_nint = -1;
    CG_CUDA_TRY(ctx->tc_poly.ensure((size_t)total * sizeof(TcPoly)));
    k_ptc_poly_int<<<ceil_div(total, 128), 128, 0, st>>>(ctx->poly.as<double>(), total, ctx->tc_poly.as<TcPoly>());
    count_launch();
    CG_CUDA_TRY(cudaGetLastError());
    CG_CUDA_TRY(cudaStreamSynchronize(st));  // other streams' calls may read the table next
    ctx->tc_poly_lmax = ctx->poly_lmax;
    ctx->tc_poly_nint = ctx->poly_nint;
    return CATANA_OK;
}

}  // namespace

// nmax: the table position k r / dx has at most 27 integer bits; rmax: k / dx stays inside FP64
bool plain_tc_takes(const DeviceContext *ctx, int lmax, int nmax, double rmax) {
    return ctx->cc_major == 10 && ctx->cc_minor == 3 && lmax <= TC_LMAX && nmax >= 1 && nmax <= 4096 && rmax > 1e-100 &&
           rmax < 1e100;
}

// A term is held to 2^-55 of its slab's bound, which goes with the slab's heaviest weight.  Where the heavy points
// add little to a mode -- they lie near a pole and m is high, or where j_l is still small -- a mode has only the
// light ones' terms, with as many bits less as they are lighter; FP64 held them all.  Up to eight bits, 2^-47 of
// such a mode's terms (7e-15), stay inside the errors that both paths have from their recurrences (5e-15 to 1e-14
// of f); a catalog whose weights differ by more takes the FP64 path.
bool plain_tc_holds(const WeightRange &wr) { return !(wr.hi > 256.0 * wr.lo); }

double plain_tc_blocks(int lmax, int nmax) {
    const double full = lmax / 64, rest = lmax - 64.0 * full;
    return (32.0 * full * (full + 1.0) + rest * (full + 1.0)) * ((nmax + 63) / 64);
}

// Few points with many radial orders, and catalogs of a few levels, are the FP64 path's: a CTA of the tensor-core
// kernel walks its blocks of 64 complex m and 64 radial orders one after the other, 11 to 15 us each (5 to 7 with
// one or two column steps), where the FP64 path has a CTA for each, and takes 35 us a level below l = 32 and 89
// above it, or its FP64 work.  Microseconds, fitted to 742 calls (l 1 to 512, n 1 to 3000, 1 to 8192 points, the
// three j_l modes): the path chosen is at most 1.2 times slower than the other, in all but 13 of them within 5%.
// For instance, tensor cores / FP64: 100 points, n 200: l 8 404 / 269, l 100 7405 / 7334, l 300 43400 / 26200; n
// 1000: l 24 6340 / 1070, l 128 48300 / 10300, with 4000 points 70100 / 178000; n 64, l 512 33400 / 44900; l 1, n
// 16 81 / 44, l 8 120 / 184.
bool plain_tc_pays(int64_t npoints, int lmax, int nmax, JlMode jl) {
    const bool few = nmax <= 32, exact = jl == JL_MODE_EXACT;
    const double n = (double)npoints, l = lmax, values = n * nmax * l;
    const double tc = 68.0 + plain_tc_blocks(lmax, nmax) * ((few ? 5.4 : 11.0) + (npoints >= 32 ? 1.5 : 0.0) + 4.9e-4 * n) +
                      (exact ? values * (5.6e-5 + 6.1e-6 * l) : 0.0);
    double base = (few ? 22.0 : 35.0) * std::min(lmax, 32) + (few ? 80.0 : 89.0) * std::max(lmax - 32, 0);
    if (jl == JL_MODE_POLY) base += 6.0 * l;
    if (exact) base += 13.0 * l * l * std::min(nmax, 64) / 64.0 * (npoints < 32 ? 0.28 : 1.0);
    const double work = n * 64.0 * ((nmax + 63) / 64) * l * (6.2e-5 + 2.4e-6 * (l + 1.0)) +
                        (exact ? values * 3.4e-5 * l : 0.0);
    return tc < 23.0 + std::sqrt(std::sqrt(base * base * base * base + work * work * work * work));
}

std::atomic<uint64_t> g_plain_stall_ns{0};

namespace {

// CATANA_ERR_NOMEM: nothing has been added, and the caller has another path.
// pix == nullptr: points_dev are npoints x 3; otherwise the pixelized catalog.  "Points" below are what the main
// kernel takes as such: the catalog's points, or a pixelized one's entries.
catana_status_t tc_accumulate(DeviceContext *ctx, const double *points_dev, const double *weights_dev,
                              const PixelCatalog *pix, int64_t nall, int lmax, int nmax, double rmax, JlMode jl,
                              double rtop, const double *kln_dev, double *f_acc_dev, int *err_dev, cudaStream_t st) {
    // the test hook (catana_gpu_test_plain_stall) arms one run
    const uint64_t stall_ns = g_plain_stall_ns.exchange(0);
    const bool lerp = jl == JL_MODE_LERP, fused = lerp && !pix;  // fused: the main kernel evaluates j_l itself
    int64_t npoints = nall;  // a pixelized catalog's entries, once they are counted
    catana_status_t s = ensure_tc_coefs(ctx, lmax, st);
    if (s != CATANA_OK) return s;
    if (lerp) {
        s = ensure_tc_tables(ctx, lmax, nmax, st);
        if (s != CATANA_OK) return s;
    }
    if (!ctx->attr_tc) {
        CG_CUDA_TRY(cudaFuncSetAttribute(k_ptc_main<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
        CG_CUDA_TRY(cudaFuncSetAttribute(k_ptc_main<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
        ctx->attr_tc = true;
    }
    const int lmp = (lmax + 3) & ~3;
    if (jl == JL_MODE_POLY) {
        s = ensure_tc_poly(ctx, st);
        if (s != CATANA_OK) return s;
    }
    // 2^er > 4 rmax: radii at or past 4 rmax lie outside the table of l = 0 whatever nmax; rtop, the largest
    // radius, where the caller knows it
    const int er = std::max(ilogb(rmax) + 3, rtop > 0.0 ? ilogb(rtop) + 1 : -1000);
    const double rlim = lerp ? ldexp(1.0, er) : INFINITY;
    // A pixelized catalog is sorted into entries first, in the workspace of the HEALPix calls (which end before they
    // return): [sort scratch][radii][ring phases][TcCall]
    TcPixels px = {};
    const uint32_t *entries = nullptr;
    const uint64_t *entry_r = nullptr;
    TcCall *call = nullptr;
    if (pix) {
        const size_t kb = tc_al((size_t)nall * 4), hb = tc_al(radix_hist_words(nall) * 4), rb = tc_al((size_t)nall * 8);
        const size_t phb = tc_al((size_t)pix->nrings * lmax * sizeof(double2));
        CG_CUDA_TRY(ctx->hp_ws.ensure(4 * kb + hb + rb + phb + 256));
        char *hs = ctx->hp_ws.as<char>();
        uint32_t *keys = reinterpret_cast<uint32_t *>(hs), *perm = reinterpret_cast<uint32_t *>(hs + kb);
        uint64_t *rint = reinterpret_cast<uint64_t *>(hs + 4 * kb + hb);
        double2 *ph = reinterpret_cast<double2 *>(hs + 4 * kb + hb + rb);
        call = reinterpret_cast<TcCall *>(hs + 4 * kb + hb + rb + phb);
        CG_CUDA_TRY(cudaMemsetAsync(call, 0, sizeof(TcCall), st));
        k_ptc_ring_phases<<<ceil_div((int64_t)pix->nrings * lmax, 128), 128, 0, st>>>(pix->ring_phi, pix->nrings, lmax, ph);
        px.r = pix->r;
        px.offs = pix->offs;
        px.npix = pix->npix;
        px.nrings = pix->nrings;
        px.lmax = lmax;
        px.conj = pix->conj ? 1 : 0;
        px.ring_start = pix->ring_start;
        px.ring_pix = pix->ring_pix;
        px.ring_x = pix->ring_x;
        px.ring_ph = ph;
        px.tw = pix->tw;
        px.tw_off = pix->tw_off;
        k_ptc_cells<<<ceil_div(nall, 256), 256, 0, st>>>(px, nall, 1.0 / rmax, er, lerp ? 1 : 0, rlim, keys, perm, rint,
                                                         call, err_dev);
        count_launch(2);
        CG_CUDA_TRY(cudaGetLastError());
        unsigned long long cells = 0;
        CG_CUDA_TRY(cudaMemcpyAsync(&cells, &call->count, sizeof(cells), cudaMemcpyDeviceToHost, st));
        s = radix_sort_pairs(keys, perm, reinterpret_cast<uint32_t *>(hs + 2 * kb),
                             reinterpret_cast<uint32_t *>(hs + 3 * kb), nall, 16,
                             reinterpret_cast<uint32_t *>(hs + 4 * kb), st);
        if (s != CATANA_OK) return s;
        CG_CUDA_TRY(cudaStreamSynchronize(st));
        npoints = (int64_t)cells;
        entries = perm;
        entry_r = rint;
    }
    // Points per pass: the rows and phases (32 B per point and m) stay under 4 GB, the J of one level (8 B per point
    // and radial order) under 2 GB, and so do the sums of more slabs than there are SMs.  The levels of a launch go by
    // their sums, 256 MB (they are read back at once and mostly hit L2), and their J, 2 GB.  Where that cannot be had
    // everything is cut to a quarter, and again, as long as a pass gives every SM a tile; nothing is allocated after.
    const double slab_bytes = 16.0 * lmax * nmax;  // of the largest level
    double scale = 1.0;
    int64_t chunk;
    // slabs: at most TC_SLAB_TILES tiles (the 64-bit sums' resolution), a whole number of waves
    auto slab_tiles = [&](int tiles) {
        const int waves = ceil_div(tiles, (int64_t)ctx->sm_count * TC_SLAB_TILES);
        return ceil_div(tiles, (int64_t)ctx->sm_count * waves);
    };
    // workspace: [perm and sort scratch][records][rows][phases][slabs][maxima][TcCall]
    size_t kb, hb, o_rint, o_rabs, o_xs, o_rows, o_ph, o_sl, o_mx, o_call;
    for (;; scale *= 0.25) {
        const double slabs_c = std::max((double)ctx->sm_count, scale * 2e9 / slab_bytes);
        double fit = std::min(scale * 4e9 / (32.0 * lmp), slabs_c * TC_SLAB_TILES * TC_KT);
        if (!fused) fit = std::min(fit, scale * 2e9 / (8.0 * nmax));
        chunk = std::min(npoints, std::max<int64_t>(TC_KT, (int64_t)fit / TC_KT * TC_KT));
        const int tiles = ceil_div(chunk, TC_KT);
        const size_t np = (size_t)tiles * TC_KT;
        kb = pix ? 0 : tc_al(np * 4), hb = pix ? 0 : tc_al(radix_hist_words((int64_t)np) * 4);
        o_rint = 4 * kb + hb, o_rabs = o_rint + tc_al(np * 8), o_xs = o_rabs + tc_al(np * 8);
        o_rows = o_xs + tc_al(np * 16), o_ph = o_rows + tc_al(2 * np * lmp * 8), o_sl = o_ph + tc_al(np * lmp * 16);
        // a last pass of fewer points may have more slabs, up to this many
        const int slabs = std::min(tiles, ctx->sm_count * ceil_div(tiles, (int64_t)ctx->sm_count * TC_SLAB_TILES));
        o_mx = o_sl + tc_al((size_t)slabs * sizeof(TcSlab)), o_call = o_mx + tc_al((size_t)slabs * 3 * TC_LMAX * 4);
        const double sums = std::max(slab_bytes * slabs, std::min(scale * 256e6, 0.5 * (lmax + 1) * slab_bytes * slabs));
        const double ntab = std::min(sums, slab_bytes * slabs);
        const double jl = fused ? 0.0 : 8.0 * np * nmax;
        cudaError_t e = ctx->tc_ws.ensure(o_call + 256);
        if (e == cudaSuccess) e = ctx->partial.ensure((size_t)(sums + ntab) + 512);
        if (e == cudaSuccess) e = ctx->tc_jarr.ensure((size_t)std::max(jl, std::min(scale * 2e9, jl * lmax)));
        if (e == cudaSuccess) break;
        const bool again = e == cudaErrorMemoryAllocation && (chunk > (int64_t)ctx->sm_count * TC_KT || scale == 1.0);
        if (!again) CG_CUDA_TRY(e);
    }
    char *ws = ctx->tc_ws.as<char>();
    uint32_t *keys = reinterpret_cast<uint32_t *>(ws), *perm = reinterpret_cast<uint32_t *>(ws + kb);
    uint32_t *tk = reinterpret_cast<uint32_t *>(ws + 2 * kb), *tv = reinterpret_cast<uint32_t *>(ws + 3 * kb);
    uint32_t *hist = reinterpret_cast<uint32_t *>(ws + 4 * kb);
    TcSlab *slabs = reinterpret_cast<TcSlab *>(ws + o_sl);
    if (!pix) {
        call = reinterpret_cast<TcCall *>(ws + o_call);
        CG_CUDA_TRY(cudaMemsetAsync(call, 0, sizeof(TcCall), st));
    }
    for (int64_t c0 = 0; c0 < npoints; c0 += chunk) {
        const int64_t nc = std::min(chunk, npoints - c0);
        const int tiles = ceil_div(nc, TC_KT);
        const int tslab = slab_tiles(tiles), nslabs = ceil_div(tiles, tslab);
        // warps per CTA: eight, or as few as still give every SM one (the FP64 pipe, one an SM, bounds both
        // kernels: 445 points, l 10: 17 us by eight, 11 so)
        const int pw = std::max(1, std::min(8, tiles * ceil_div(lmp, 8) / ctx->sm_count));
        const dim3 pg(ceil_div(tiles, pw), ceil_div(lmp, 8));
        uint64_t *rint_d = reinterpret_cast<uint64_t *>(ws + o_rint);
        double *rabs_d = reinterpret_cast<double *>(ws + o_rabs);
        double2 *xs_d = reinterpret_cast<double2 *>(ws + o_xs);
        ulonglong2 *ph_d = reinterpret_cast<ulonglong2 *>(ws + o_ph);
        uint2 *cell = reinterpret_cast<uint2 *>(ws + o_rabs);
        if (pix) {
            k_ptc_pixels<<<pg, 32 * pw, 0, st>>>(px, entries + c0, nc, tiles, lmp, cell, xs_d, ph_d);
            k_ptc_cell_slabs<<<nslabs, 256, 0, st>>>(px, cell, nc, (int64_t)tslab * TC_KT, rlim, slabs, call);
        } else {
            const double *pts = points_dev + 3 * c0, *w = weights_dev ? weights_dev + c0 : nullptr;
            // Neighbours share cells of the j_l table and slabs take a bound each.  A tile of 32 of few points
            // spans more than one of 256 steps anyway: one pass of the sort instead of two.
            const int bits = nc <= 8192 ? 8 : 16;
            k_ptc_keys<<<ceil_div(nc, 256), 256, 0, st>>>(pts, nc, 1.0 / rmax, bits, keys, perm);
            count_launch();
            s = radix_sort_pairs(keys, perm, tk, tv, nc, bits, hist, st);
            if (s != CATANA_OK) return s;
            k_ptc_slabs<<<nslabs, 256, 0, st>>>(pts, w, perm, nc, (int64_t)tslab * TC_KT, rlim, slabs, call);
            k_ptc_points<<<pg, 32 * pw, 0, st>>>(pts, w, perm, nc, tiles, tslab, lmp, slabs, er, lerp ? 1 : 0, rlim,
                                                 rint_d, rabs_d, xs_d, ph_d, call, err_dev);
        }
        count_launch(2);
        CG_CUDA_TRY(cudaGetLastError());
        TcArgs a;
        a.nmax = nmax;
        a.lmp = lmp;
        a.tiles = tiles;
        a.tslab = tslab;
        a.phase = reinterpret_cast<const ulonglong2 *>(ws + o_ph);
        a.rows = reinterpret_cast<double *>(ws + o_rows);
        a.rint = pix ? entry_r : reinterpret_cast<const uint64_t *>(ws + o_rint);
        a.xs = reinterpret_cast<const double2 *>(ws + o_xs);
        a.slab = slabs;
        a.coef = ctx->tc_coef.as<double2>();
        a.npts = 1000 * nmax;
        a.maxq = reinterpret_cast<uint32_t *>(ws + o_mx);
        a.err = err_dev;
        a.wait_ns = stall_ns ? stall_ns : TC_WAIT_NS;
        a.stall = stall_ns ? 1 : 0;
        a.call = call;
        a.tab = nullptr;
        const double *dxinv = nullptr;
        if (lerp) {
            if (fused) a.tab = ctx->tc_tab.as<double2>();
            dxinv = reinterpret_cast<const double *>(ctx->tc_tab.as<char>() + ctx->tc_tab_off);
        }
        for (int l0 = 0; l0 < lmax;) {
            int l1 = l0 + 1;
            auto pdoubles = [&](int e) { return (int64_t)nmax * ((int64_t)e * (e + 1) - (int64_t)l0 * (l0 + 1)); };
            const double jbytes = fused ? 0.0 : 8.0 * tiles * TC_KT * nmax;
            while (l1 < lmax && pdoubles(l1 + 1) * 8.0 * nslabs < scale * 256e6 &&
                   jbytes * (l1 + 1 - l0) < scale * 2e9)
                ++l1;
            a.l0 = l0;
            a.l1 = l1;
            a.pslab = pdoubles(l1);
            const size_t pb = tc_al((size_t)a.pslab * nslabs * 8);
            a.partial = ctx->partial.as<double>();
            uint4 *ntab = reinterpret_cast<uint4 *>(ctx->partial.as<char>() + pb);
            a.ntab = ntab;
            k_ptc_ntab<<<dim3(nslabs, ceil_div((int64_t)(l1 - l0) * nmax, 128)), 128, 0, st>>>(
                slabs, kln_dev, dxinv, dxinv ? dxinv + ctx->tc_tab_lmax : nullptr, l0, l1 - l0, nmax, er, ntab, err_dev);
            count_launch();
            a.jarr = nullptr;
            if (!fused) {
                const int64_t cnt = (int64_t)(l1 - l0) * tiles * nmax * TC_KT;
                uint64_t *ja = ctx->tc_jarr.as<uint64_t>();
                TcJ j;
                j.r = pix ? pix->r : reinterpret_cast<const double *>(ws + o_rabs);
                j.cell = cell;
                j.tab = ctx->tc_tab.as<double2>();
                j.npts = a.npts;
                j.kln = kln_dev;
                j.rint = a.rint;
                j.ntab = ntab;
                j.l0 = l0;
                j.nl = l1 - l0;
                j.nmax = nmax;
                j.tiles = tiles;
                j.tslab = tslab;
                j.er = er;
                j.out = ja;
                if (pix && lerp)
                    k_ptc_jl_cells<<<ceil_div((int64_t)(l1 - l0) * tiles * ((nmax + JC_N - 1) / JC_N), 8), 256, 0, st>>>(j);
                else if (pix)
                    k_ptc_jl_cells_exact<<<ceil_div(cnt, 256), 256, 0, st>>>(j);
                else if (jl == JL_MODE_POLY)
                    k_ptc_jl_poly<<<ceil_div(cnt, 256), 256, 0, st>>>(j, ctx->tc_poly.as<TcPoly>(), ctx->tc_poly_nint,
                                                                      err_dev);
                else
                    k_ptc_jl_exact<<<ceil_div(cnt, 256), 256, 0, st>>>(j);
                count_launch();
                CG_CUDA_TRY(cudaGetLastError());
                a.jarr = ja;
            }
            prof_begin(st);
            if (fused) k_ptc_main<true><<<nslabs, TC_THREADS, TC_SMEM, st>>>(a);
            else k_ptc_main<false><<<nslabs, TC_THREADS, TC_SMEM, st>>>(a);
            prof_end(st, 2.0 * (double)nc * (double)pdoubles(l1));
            k_ptc_reduce<<<dim3(std::min(64, ceil_div((int64_t)l1 * nmax, 32)), l1 - l0), 256, 0, st>>>(
                a.partial, a.pslab, nslabs, l0, nmax, kln_dev, call, reinterpret_cast<double2 *>(f_acc_dev));
            count_launch(2);
            CG_CUDA_TRY(cudaGetLastError());
            l0 = l1;
        }
    }
    return CATANA_OK;
}

}  // namespace

catana_status_t plain_tc_accumulate(DeviceContext *ctx, const double *points_dev, const double *weights_dev, int64_t npoints,
                                    int lmax, int nmax, double rmax, JlMode jl, double rtop, const double *kln_dev,
                                    double *f_acc_dev, int *err_dev, cudaStream_t st) {
    return tc_accumulate(ctx, points_dev, weights_dev, nullptr, npoints, lmax, nmax, rmax, jl, rtop, kln_dev, f_acc_dev,
                         err_dev, st);
}

catana_status_t plain_tc_pixels(DeviceContext *ctx, const PixelCatalog &pix, int64_t npoints, int lmax, int nmax,
                                double rmax, JlMode jl, const double *kln_dev, double *f_acc_dev, int *err_dev,
                                cudaStream_t st) {
    return tc_accumulate(ctx, nullptr, nullptr, &pix, npoints, lmax, nmax, rmax, jl, 0.0, kln_dev, f_acc_dev, err_dev, st);
}

}  // namespace catana_gpu

extern "C" catana_status_t catana_gpu_test_plain_stall(uint32_t wait_us) {
    if (wait_us < 1 || wait_us > 1000000) {
        catana_gpu::set_error("test_plain_stall: wait_us must be in [1, 1000000]");
        return CATANA_ERR_ARG;
    }
    catana_gpu::g_plain_stall_ns.store((uint64_t)wait_us * 1000ull);
    return CATANA_OK;
}
