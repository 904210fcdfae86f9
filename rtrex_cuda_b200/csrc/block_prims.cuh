// Exclusive scan and stable radix sort by one block of 1,024 threads: the small
// cases of primitives.cu, and steps of kernels that do the whole set-up of a small
// stage in one launch.  The caller synchronises the block before and after.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace rtr {

constexpr int kRadixBits = 8;
constexpr int kBins = 1 << kRadixBits;
constexpr int kOneBlock = 1024;
constexpr int kOneItems = 16;
constexpr int64_t kScanOne = (int64_t)kOneBlock * kOneItems;

// n <= kScanOne; s_warp: 32 elements of shared memory.
template <typename T>
__device__ __forceinline__ void scan_one(const T* in, T* out, int n, T* total, T* s_warp)
{
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    // warp w holds [w * per, (w + 1) * per), 32 elements at a time
    const int per = ((n + 31) / 32 + 31) / 32 * 32, w0 = warp * per;
    T acc = 0;
    for (int b = 0; b < per; b += 32) {
        const int i = w0 + b + lane;
        acc += i < n ? in[i] : T(0);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) s_warp[warp] = acc;
    __syncthreads();
    T run = 0, all = 0;
    for (int w = 0; w < 32; ++w) {
        const T x = s_warp[w];
        run += w < warp ? x : T(0);
        all += x;
    }
    for (int b = 0; b < per; b += 32) {
        const int i = w0 + b + lane;
        const T v = i < n ? in[i] : T(0);
        T x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (i < n) out[i] = run + x - v;
        run += __shfl_sync(0xffffffffu, x, 31);
    }
    if (t == 0 && total) *total = all;
}

// Stable rank of a key's digit inside its warp's run: the number of earlier keys
// of the warp with the same digit (cnt[d], advanced here; d == kBins: no key).
__device__ __forceinline__ unsigned warp_rank(uint32_t* cnt, unsigned d, int lane)
{
    const unsigned peers = __match_any_sync(0xffffffffu, d);
    const unsigned r = __popc(peers & ((1u << lane) - 1u));
    const unsigned before = cnt[d];
    __syncwarp();
    if (r == 0) cnt[d] = before + __popc(peers);
    __syncwarp();
    return before + r;
}

// Exclusive scan of one value per thread over the first 256 threads of a block.
__device__ __forceinline__ uint32_t bins_exclusive_scan(uint32_t v, uint32_t* s_warp)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31 && warp < kBins / 32) s_warp[warp] = x;
    __syncthreads();
    uint32_t pre = 0;
    for (int w = 0; w < kBins / 32; ++w) pre += w < warp ? s_warp[w] : 0u;
    __syncthreads();
    return pre + x - v;
}

// All digits of up to kSortOne keys in shared memory, one block.  Each warp holds a
// run of the keys; per digit: the runs' histograms, their offsets, the scatter.
constexpr int kSortOne = 8192;
constexpr int kSortWarps = 32;

struct SortOneSmem {
    uint64_t key[2][kSortOne];
    uint32_t cnt[kSortWarps][kBins + 1];
    uint32_t warp[kBins / 32];
};

__device__ __forceinline__ void sort_one(SortOneSmem& S, const uint64_t* in, uint64_t* out, int n, int lo, int hi)
{
    constexpr int T = 32 * kSortWarps;
    constexpr int kMax = kSortOne / T;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int rounds = (n + T - 1) / T;  // keys per thread
    const int w0 = warp * 32 * rounds;   // this warp's run
    for (int i = t; i < n; i += T) S.key[0][i] = in[i];
    __syncthreads();
    int cur = 0;
    for (int shift = lo; shift < hi; shift += kRadixBits) {
        for (int i = t; i < kSortWarps * (kBins + 1); i += T) (&S.cnt[0][0])[i] = 0;
        __syncthreads();
        uint64_t k[kMax];
        unsigned r[kMax];
#pragma unroll
        for (int q = 0; q < kMax; ++q) {
            if (q < rounds) {
                const int i = w0 + q * 32 + lane;
                const bool valid = i < n;
                k[q] = valid ? S.key[cur][i] : 0ull;
                const unsigned d = valid ? (unsigned)((k[q] >> shift) & (kBins - 1)) : (unsigned)kBins;
                r[q] = warp_rank(S.cnt[warp], d, lane);
            }
        }
        __syncthreads();
        // digit t: the warps' counts become offsets
        uint32_t sum = 0;
        if (t < kBins)
            for (int w = 0; w < kSortWarps; ++w) {
                const uint32_t c = S.cnt[w][t];
                S.cnt[w][t] = sum;
                sum += c;
            }
        const uint32_t base = bins_exclusive_scan(t < kBins ? sum : 0u, S.warp);
        if (t < kBins)
            for (int w = 0; w < kSortWarps; ++w) S.cnt[w][t] += base;
        __syncthreads();
#pragma unroll
        for (int q = 0; q < kMax; ++q) {
            const int i = w0 + q * 32 + lane;
            if (q < rounds && i < n) {
                const unsigned d = (unsigned)((k[q] >> shift) & (kBins - 1));
                S.key[cur ^ 1][S.cnt[warp][d] + r[q]] = k[q];
            }
        }
        cur ^= 1;
        __syncthreads();
    }
    for (int i = t; i < n; i += T) out[i] = S.key[cur][i];
}

}  // namespace rtr
