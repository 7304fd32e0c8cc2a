// sort.cu -- stable LSD radix sort of (uint32 key, uint32 index) pairs on the GPU.
//
// Used to group points: by HEALPix pixel for the binned catalog (the reference
// appends radii to per-pixel vectors in point order, PixelizedPointContainer.cpp:27-30,
// so the sort must be stable) and by quantised radius for the split form (points
// with nearly equal r share j_l table intervals, which turns the shared-memory table
// reads into broadcasts).
//
// One pass per 8-bit digit:
//   k_radix_hist     per-tile digit histogram (tile = up to 4096 consecutive pairs)
//   k_radix_scan     exclusive scan of the (digit-major, tile-minor) histogram
//   k_radix_scatter  each tile re-reads its pairs in order, 256 at a time, ranks equal
//                    digits with __match_any_sync within a warp and with per-warp
//                    counts across warps, and scatters -- a stable, deterministic order.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "common.cuh"

namespace catana_gpu {

namespace {

constexpr int RS_THREADS = 256;
constexpr int RS_ROUNDS = 16;  // most rounds of 256 pairs per tile
constexpr int RS_WARPS = RS_THREADS / 32;

__global__ void k_radix_hist(const uint32_t *__restrict__ keys, int64_t n, int shift, uint32_t *__restrict__ hist,
                             int ntiles, int tile) {
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * tile;
    for (int k = threadIdx.x; k < tile; k += RS_THREADS) {
        const int64_t i = base + k;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[(size_t)threadIdx.x * ntiles + blockIdx.x] = h[threadIdx.x];
}

// Single-CTA exclusive scan of count entries: 1024 threads take 16384 consecutive words a round,
// sixteen each as four 16-byte loads, and load the next round's words before they scan this one's,
// so a round costs one scan and not a trip to memory (62.7k words, the histogram of 1M pairs: 16 us;
// with a contiguous segment per thread, read word by word twice, 61).
constexpr int SC_PER = 16;
__global__ void __launch_bounds__(1024) k_radix_scan(uint32_t *__restrict__ data, int64_t count) {
    __shared__ uint32_t part[2][32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const bool vec = (reinterpret_cast<uintptr_t>(data) & 15) == 0;
    auto load = [&](int64_t base, uint32_t (&v)[SC_PER]) {
        const int64_t i = base + (int64_t)SC_PER * t;
        if (vec && i + SC_PER <= count) {
#pragma unroll
            for (int k = 0; k < SC_PER; k += 4) {
                const uint4 q = *reinterpret_cast<const uint4 *>(data + i + k);
                v[k] = q.x;
                v[k + 1] = q.y;
                v[k + 2] = q.z;
                v[k + 3] = q.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < SC_PER; ++k) v[k] = i + k < count ? data[i + k] : 0u;
        }
    };
    uint32_t v[SC_PER], nx[SC_PER];
    load(0, v);
    uint32_t carry = 0;
    int par = 0;
    for (int64_t base = 0; base < count; base += 1024 * SC_PER, par ^= 1) {
        load(base + 1024 * SC_PER, nx);  // words the others have not written yet: a later round's
        uint32_t s = 0;
#pragma unroll
        for (int k = 0; k < SC_PER; ++k) {  // exclusive within the thread
            const uint32_t x = v[k];
            v[k] = s;
            s += x;
        }
        uint32_t inc = s;  // inclusive over the warp's threads
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += y;
        }
        if (lane == 31) part[par][warp] = inc;
        __syncthreads();  // two buffers: the next round's writes come after the next barrier's reads
        uint32_t wsum = part[par][lane];  // every warp scans the 32 warp sums
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, wsum, o);
            if (lane >= o) wsum += y;
        }
        const uint32_t before = warp ? __shfl_sync(0xffffffffu, wsum, warp - 1) : 0u;
        const uint32_t add = carry + before + inc - s;
        carry += __shfl_sync(0xffffffffu, wsum, 31);
        const int64_t i = base + (int64_t)SC_PER * t;
        if (vec && i + SC_PER <= count) {
#pragma unroll
            for (int k = 0; k < SC_PER; k += 4)
                *reinterpret_cast<uint4 *>(data + i + k) =
                    make_uint4(v[k] + add, v[k + 1] + add, v[k + 2] + add, v[k + 3] + add);
        } else {
#pragma unroll
            for (int k = 0; k < SC_PER; ++k)
                if (i + k < count) data[i + k] = v[k] + add;
        }
#pragma unroll
        for (int k = 0; k < SC_PER; ++k) v[k] = nx[k];
    }
}

__global__ void k_radix_scatter(const uint32_t *__restrict__ keys, const uint32_t *__restrict__ vals, int64_t n,
                                int shift, const uint32_t *__restrict__ offs, int ntiles,
                                uint32_t *__restrict__ keys_out, uint32_t *__restrict__ vals_out, int tile) {
    __shared__ uint32_t base[256];
    __shared__ uint32_t wcnt[RS_WARPS][256];
    const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
    base[t] = offs[(size_t)t * ntiles + blockIdx.x];
    for (int w = 0; w < RS_WARPS; ++w) wcnt[w][t] = 0;
    __syncthreads();
    const uint32_t lt_mask = (1u << lane) - 1u;
    const int64_t tile0 = (int64_t)blockIdx.x * tile;
    for (int r = 0; r < tile / RS_THREADS; ++r) {
        const int64_t i = tile0 + (int64_t)r * RS_THREADS + t;
        const bool valid = i < n;
        uint32_t key = 0, val = 0, d = 0xFFFFFFFFu;  // invalid lanes form their own group
        if (valid) {
            key = keys[i];
            val = vals[i];
            d = (key >> shift) & 255u;
        }
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
        const uint32_t rank = __popc(peers & lt_mask);
        if (valid && rank == 0) wcnt[warp][d] = __popc(peers);
        __syncthreads();
        if (valid) {
            uint32_t before = 0;
            for (int w = 0; w < warp; ++w) before += wcnt[w][d];
            const uint32_t dst = base[d] + before + rank;
            keys_out[dst] = key;
            vals_out[dst] = val;
        }
        __syncthreads();
        uint32_t tot = 0;
        for (int w = 0; w < RS_WARPS; ++w) {
            tot += wcnt[w][t];
            wcnt[w][t] = 0;
        }
        base[t] += tot;
        __syncthreads();
    }
}

}  // namespace

// In-place exclusive scan of count uint32 words (single CTA; counts up to a few
// million entries).
catana_status_t scan_u32(uint32_t *data, int64_t count, cudaStream_t st) {
    if (count <= 0) return CATANA_OK;
    k_radix_scan<<<1, 1024, 0, st>>>(data, count);
    count_launch();
    CG_CUDA_TRY(cudaGetLastError());
    return CATANA_OK;
}

namespace {
// Pairs per tile: a tile's rounds run one after the other (1.3 us each in the scatter), so fewer than
// 262144 pairs take as few rounds as leave at most 64 tiles, whose histogram the scan takes in one round.
// 5000 pairs, a pass: 35 us by tiles of 4096, 12 so.
int radix_tile(int64_t n) {
    const int64_t rounds = (n + 64 * RS_THREADS - 1) / (64 * RS_THREADS);
    return RS_THREADS * (int)std::min<int64_t>(RS_ROUNDS, std::max<int64_t>(1, rounds));
}
}  // namespace

size_t radix_hist_words(int64_t n) {
    return (size_t)256 * (size_t)std::max<int64_t>(64, (n + RS_ROUNDS * RS_THREADS - 1) / (RS_ROUNDS * RS_THREADS));
}

// Sorts (keys, vals) by the low `key_bits` bits of the keys, stably.  The result
// ends in (keys, vals); tmp_keys / tmp_vals are scratch of n entries; hist_scratch
// holds radix_hist_words(n) words.
catana_status_t radix_sort_pairs(uint32_t *keys, uint32_t *vals, uint32_t *tmp_keys, uint32_t *tmp_vals, int64_t n,
                                 int key_bits, uint32_t *hist_scratch, cudaStream_t st) {
    if (n <= 1) return CATANA_OK;
    const int tile = radix_tile(n), ntiles = (int)((n + tile - 1) / tile);
    uint32_t *ka = keys, *va = vals, *kb = tmp_keys, *vb = tmp_vals;
    int passes = 0;
    for (int shift = 0; shift < key_bits; shift += 8, ++passes) {
        k_radix_hist<<<ntiles, RS_THREADS, 0, st>>>(ka, n, shift, hist_scratch, ntiles, tile);
        k_radix_scan<<<1, 1024, 0, st>>>(hist_scratch, (int64_t)256 * ntiles);
        k_radix_scatter<<<ntiles, RS_THREADS, 0, st>>>(ka, va, n, shift, hist_scratch, ntiles, kb, vb, tile);
        count_launch(3);
        CG_CUDA_TRY(cudaGetLastError());
        uint32_t *t;
        t = ka;
        ka = kb;
        kb = t;
        t = va;
        va = vb;
        vb = t;
    }
    if (passes & 1) {  // result sits in the scratch arrays: copy back
        CG_CUDA_TRY(cudaMemcpyAsync(keys, ka, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
        CG_CUDA_TRY(cudaMemcpyAsync(vals, va, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
    }
    return CATANA_OK;
}

}  // namespace catana_gpu
