// Exclusive scan and stable LSD radix sort, sm_100a.
//
// The small forms take one launch each (a decomposition of a small graph is
// bound by its launches): up to 16,384 elements are scanned, and up to 8,192
// keys sorted over all their digits, by one block.  Larger scans are
// reduce-then-scan; a larger sort takes one pass over the keys for all digits'
// histograms and one per digit, whose tiles find their offsets by decoupled
// look-back (each key is read and written once per digit; a separate histogram
// and three scan launches per digit read them twice).  Measured on B200: the
// decomposition of a 1,003-edge graph 2.38 -> 1.89 ms (166 -> 69 launches); CSR
// builds of 500 / 20,000 / 926,000 / 5,000,000 edges 0.22 -> 0.16, 0.28 -> 0.22,
// 1.30 -> 1.16, 8.29 -> 7.50 ms (the rest is the copy in and the CSR's own passes).
#include "primitives.cuh"
#include "block_prims.cuh"
#include "rtr_common.cuh"

#include <algorithm>

namespace rtr {

namespace {

constexpr int kBlock = 256;
constexpr int kItems = 8;
constexpr int kTile = kBlock * kItems;  // 2048 elements per CTA tile

template <typename T>
__device__ T block_exclusive_scan(T v, T* s_warp, T* total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kWarps = kBlock / 32;
    T x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        T y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        T w = lane < kWarps ? s_warp[lane] : T(0);
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            T y = __shfl_up_sync(0xffffffffu, w, off);
            if (lane >= off) w += y;
        }
        if (lane < kWarps) s_warp[lane] = w;
    }
    __syncthreads();
    const T prefix = warp > 0 ? s_warp[warp - 1] : T(0);
    if (total) *total = s_warp[kWarps - 1];
    __syncthreads();
    return prefix + x - v;
}

template <typename T>
__global__ void __launch_bounds__(kBlock) k_scan_reduce(const T* __restrict__ in, int64_t n, T* __restrict__ sums)
{
    __shared__ T s_warp[32];
    const int64_t base = (int64_t)blockIdx.x * kTile + (int64_t)threadIdx.x * kItems;
    T acc = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k)
        if (base + k < n) acc += in[base + k];
    T tot;
    block_exclusive_scan<T>(acc, s_warp, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// One CTA scans the per-tile sums in place (exclusive) and writes the total.
template <typename T>
__global__ void __launch_bounds__(kBlock) k_scan_top(T* __restrict__ sums, int64_t nb, T* __restrict__ total)
{
    __shared__ T s_warp[32];
    T carry = 0;
    for (int64_t start = 0; start < nb; start += kTile) {
        const int64_t base = start + (int64_t)threadIdx.x * kItems;
        T loc[kItems];
        T acc = 0;
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            loc[k] = (base + k < nb) ? sums[base + k] : T(0);
            acc += loc[k];
        }
        T tile_tot;
        T pre = block_exclusive_scan<T>(acc, s_warp, &tile_tot) + carry;
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            if (base + k < nb) sums[base + k] = pre;
            pre += loc[k];
        }
        carry += tile_tot;
    }
    if (threadIdx.x == 0 && total) *total = carry;
}

template <typename T>
__global__ void __launch_bounds__(kBlock) k_scan_down(const T* __restrict__ in, T* __restrict__ out, int64_t n,
                                                       const T* __restrict__ sums)
{
    __shared__ T s_warp[32];
    const int64_t base = (int64_t)blockIdx.x * kTile + (int64_t)threadIdx.x * kItems;
    T loc[kItems];
    T acc = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        loc[k] = (base + k < n) ? in[base + k] : T(0);
        acc += loc[k];
    }
    T pre = block_exclusive_scan<T>(acc, s_warp, nullptr) + sums[blockIdx.x];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        if (base + k < n) out[base + k] = pre;
        pre += loc[k];
    }
}

template <typename T>
__global__ void __launch_bounds__(kOneBlock) k_scan_one(const T* __restrict__ in, T* __restrict__ out, int n,
                                                        T* __restrict__ total)
{
    __shared__ T s_warp[32];
    scan_one(in, out, n, total, s_warp);
}

// Kernels launched by this thread's scans and sorts since the last call of take_primitive_launches.
thread_local int64_t t_launches = 0;

template <typename T>
int scan_impl(const T* d_in, T* d_out, int64_t n, T* d_total, T* temp, cudaStream_t s)
{
    if (n <= 0) {
        if (d_total) RTR_CUDA_TRY(cudaMemsetAsync(d_total, 0, sizeof(T), s));
        return RTR_OK;
    }
    if (n <= kScanOne) {
        k_scan_one<T><<<1, kOneBlock, 0, s>>>(d_in, d_out, (int)n, d_total);
        t_launches += 1;
        RTR_CUDA_TRY(cudaGetLastError());
        return RTR_OK;
    }
    const int64_t nb = (n + kTile - 1) / kTile;
    k_scan_reduce<T><<<(unsigned)nb, kBlock, 0, s>>>(d_in, n, temp);
    k_scan_top<T><<<1, kBlock, 0, s>>>(temp, nb, d_total);
    k_scan_down<T><<<(unsigned)nb, kBlock, 0, s>>>(d_in, d_out, n, temp);
    t_launches += 3;
    RTR_CUDA_TRY(cudaGetLastError());
    return RTR_OK;
}

// ---------------------------------------------------------------- radix sort

__global__ void __launch_bounds__(32 * kSortWarps) k_sort_one(const uint64_t* __restrict__ in,
                                                              uint64_t* __restrict__ out, int n, int lo, int hi)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    sort_one(*reinterpret_cast<SortOneSmem*>(smem_raw), in, out, n, lo, hi);
}

constexpr int kMaxDigits = 8;
constexpr int kPassItems = 16;
constexpr int kPassTile = kBlock * kPassItems;  // 4096 keys per tile of a digit's pass
constexpr long kLookbackLimit = 1l << 21;       // polls of an earlier tile (a second) before it is counted instead
constexpr int64_t kOneRegionFrom = (1ll << 24) + 1;  // keys from which the passes share one region of status words
constexpr int64_t kWideFrom = 1ll << 30;             // keys from which a status word is 64 bits

// Every digit's histogram in one read of the keys.
__global__ void __launch_bounds__(kBlock) k_radix_hist(const uint64_t* __restrict__ keys, int64_t n, int lo,
                                                        int digits, unsigned long long* __restrict__ hist)
{
    __shared__ uint32_t h[kMaxDigits][kBins];
    for (int i = threadIdx.x; i < digits * kBins; i += kBlock) (&h[0][0])[i] = 0;
    __syncthreads();
    for (int64_t i = blockIdx.x * (int64_t)kBlock + threadIdx.x; i < n; i += (int64_t)gridDim.x * kBlock) {
        const uint64_t k = keys[i] >> lo;
        for (int d = 0; d < digits; ++d) atomicAdd(&h[d][(k >> (d * kRadixBits)) & (kBins - 1)], 1u);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < digits * kBins; i += kBlock) {
        const uint32_t c = (&h[0][0])[i];
        if (c) atomicAdd(&hist[i], (unsigned long long)c);
    }
}

// One digit's pass (stable).  Tiles are taken in order from a counter; a tile's
// keys are ranked by warp, its digit counts published, and each digit's offset
// found by looking back over the earlier tiles (status word: 0 not yet, 1 the
// tile's own count, 2 the count through the tile, in the top two bits).  A tile
// only waits for tiles taken before it, whose blocks are running; should a wait
// run out all the same (wait_limit polls), the thread counts its digit in that
// tile's keys itself and goes on, so that no wait can end in a wrong place.
template <typename S>
__global__ void __launch_bounds__(kBlock) k_radix_pass(const uint64_t* __restrict__ keys, uint64_t* __restrict__ out,
                                                        int64_t n, int shift,
                                                        const unsigned long long* __restrict__ hist,
                                                        S* __restrict__ status, unsigned* __restrict__ next_tile,
                                                        long wait_limit)
{
    constexpr int kWarps = kBlock / 32;
    constexpr int kShift = 8 * sizeof(S) - 2;
    constexpr S kMask = ((S)1 << kShift) - 1;
    __shared__ uint64_t s_key[kPassTile];
    __shared__ uint32_t s_cnt[kWarps][kBins + 1];
    __shared__ int64_t s_base[kBins];
    __shared__ uint32_t s_warp[kBins / 32];
    __shared__ unsigned long long s_warp64[kBins / 32];
    __shared__ unsigned s_tile;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    if (t == 0) s_tile = atomicAdd(next_tile, 1u);
    for (int i = t; i < kWarps * (kBins + 1); i += kBlock) (&s_cnt[0][0])[i] = 0;
    __syncthreads();
    const int64_t tile = s_tile;
    const int64_t base = tile * kPassTile + (int64_t)warp * (32 * kPassItems);
    uint64_t k[kPassItems];
    uint32_t r[kPassItems];
#pragma unroll
    for (int q = 0; q < kPassItems; ++q) {
        const int64_t i = base + q * 32 + lane;
        k[q] = i < n ? keys[i] : 0ull;
    }
#pragma unroll
    for (int q = 0; q < kPassItems; ++q) {
        const bool valid = base + q * 32 + lane < n;
        r[q] = warp_rank(s_cnt[warp], valid ? (unsigned)((k[q] >> shift) & (kBins - 1)) : (unsigned)kBins, lane);
    }
    __syncthreads();
    // digit t: the warps' counts become offsets; publish the tile's count
    uint32_t sum = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        const uint32_t c = s_cnt[w][t];
        s_cnt[w][t] = sum;
        sum += c;
    }
    volatile S* st = status + t;
    if (tile > 0) st[tile * kBins] = ((S)1 << kShift) | (S)sum;
    const uint32_t excl = bins_exclusive_scan(sum, s_warp);
    // where the digit's keys begin
    unsigned long long h = hist[t], hx = h;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, hx, o);
        if (lane >= o) hx += y;
    }
    if (lane == 31) s_warp64[warp] = hx;
    __syncthreads();
    unsigned long long start = hx - h;
    for (int w = 0; w < warp; ++w) start += s_warp64[w];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) s_cnt[w][t] += excl;
    // the keys of earlier tiles with this digit
    S before = 0;
    for (int64_t p = tile - 1; p >= 0;) {
        const S x = st[p * kBins];
        const unsigned f = (unsigned)(x >> kShift);
        if (f == 0) {
            long spin = 0;
            bool there = false;
            while (spin++ < wait_limit && !(there = (st[p * kBins] >> kShift) != 0)) {
            }
            if (there) continue;
            const uint64_t* k0 = keys + p * kPassTile;  // an earlier tile is a whole one
            for (int i = 0; i < kPassTile; ++i) before += ((k0[i] >> shift) & (kBins - 1)) == (uint64_t)t ? 1 : 0;
            --p;
            continue;
        }
        before += x & kMask;
        if (f == 2) break;
        --p;
    }
    st[tile * kBins] = ((S)2 << kShift) | (before + (S)sum);
    s_base[t] = (int64_t)start + (int64_t)before - (int64_t)excl;
    __syncthreads();
    // through shared memory in digit order, so that the writes run along each digit
#pragma unroll
    for (int q = 0; q < kPassItems; ++q)
        if (base + q * 32 + lane < n) {
            const unsigned d = (unsigned)((k[q] >> shift) & (kBins - 1));
            s_key[s_cnt[warp][d] + r[q]] = k[q];
        }
    __syncthreads();
    const int64_t left = n - tile * kPassTile;
    const int cnt = left < kPassTile ? (int)left : kPassTile;
    for (int i = t; i < cnt; i += kBlock) {
        const uint64_t key = s_key[i];
        const int64_t at = s_base[(key >> shift) & (kBins - 1)] + i;
        if (at >= 0 && at < n) out[at] = key;
    }
}

// Tiles' status words of one pass, and how many passes keep their own (one
// clearing then serves all; a large sort clears one region before each pass).
struct RadixPlan {
    int64_t tiles, words;
    bool wide;  // 64-bit words: counts of 2^30 and more
    int64_t regions;
    RadixPlan(int64_t n, const SortForms& f)
        : tiles((n + kPassTile - 1) / kPassTile), words(tiles * kBins), wide(n >= std::min(f.wide_from, kWideFrom)),
          regions(n < f.one_region_from ? kMaxDigits : 1)
    {
    }
    size_t region_bytes() const { return (size_t)words * (wide ? 8 : 4); }
    // histograms and tile counters, then the regions
    static constexpr size_t kHead = sizeof(unsigned long long) * kMaxDigits * kBins + sizeof(unsigned) * 64;
    size_t bytes() const { return kHead + region_bytes() * (size_t)regions; }
};

}  // namespace

int64_t scan_temp_elems(int64_t n)
{
    return (n + kTile - 1) / kTile + 1;
}

int exclusive_scan_u32(const uint32_t* d_in, uint32_t* d_out, int64_t n, uint32_t* d_total, uint32_t* temp,
                       cudaStream_t s)
{
    return scan_impl<uint32_t>(d_in, d_out, n, d_total, temp, s);
}

int exclusive_scan_i64(const int64_t* d_in, int64_t* d_out, int64_t n, int64_t* d_total, int64_t* temp,
                       cudaStream_t s)
{
    return scan_impl<int64_t>(d_in, d_out, n, d_total, temp, s);
}

SortForms::SortForms() : wait_limit(kLookbackLimit), one_region_from(kOneRegionFrom), wide_from(kWideFrom) {}

size_t radix_temp_bytes(int64_t n, const SortForms& forms)
{
    // enough for any smaller n too
    if (n <= kSortOne) return 16;
    const size_t b = RadixPlan(n, forms).bytes();
    return n >= forms.one_region_from ? std::max(b, RadixPlan(forms.one_region_from - 1, forms).bytes()) : b;
}

int radix_sort_u64(uint64_t* d_keys, uint64_t* d_alt, int64_t n, int nbits, void* temp, cudaStream_t s,
                   uint64_t** sorted)
{
    return radix_sort_bits_u64(d_keys, d_alt, n, 0, nbits, temp, s, sorted);
}

int64_t take_primitive_launches()
{
    const int64_t k = t_launches;
    t_launches = 0;
    return k;
}

int radix_sort_bits_u64(uint64_t* d_keys, uint64_t* d_alt, int64_t n, int lo, int hi, void* temp, cudaStream_t s,
                        uint64_t** sorted, const SortForms& forms)
{
    *sorted = d_keys;
    if (n <= 1 || hi <= lo) return RTR_OK;
    if (n <= kSortOne) {
        const size_t smem = sizeof(SortOneSmem);
        RTR_CUDA_TRY(cudaFuncSetAttribute(k_sort_one, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_sort_one<<<1, 32 * kSortWarps, smem, s>>>(d_keys, d_alt, (int)n, lo, hi);
        t_launches += 1;
        RTR_CUDA_TRY(cudaGetLastError());
        *sorted = d_alt;
        return RTR_OK;
    }
    const RadixPlan plan(n, forms);
    const int digits = (hi - lo + kRadixBits - 1) / kRadixBits;
    unsigned long long* hist = (unsigned long long*)temp;
    unsigned* next = (unsigned*)(hist + kMaxDigits * kBins);
    unsigned char* status = (unsigned char*)temp + RadixPlan::kHead;
    const bool own = plan.regions > 1;
    RTR_CUDA_TRY(cudaMemsetAsync(temp, 0, RadixPlan::kHead + (own ? plan.region_bytes() * (size_t)digits : 0), s));
    k_radix_hist<<<grid_for(n, kBlock, 8), kBlock, 0, s>>>(d_keys, n, lo, digits, hist);
    uint64_t* src = d_keys;
    uint64_t* dst = d_alt;
    for (int d = 0; d < digits; ++d) {
        unsigned char* st = status + (own ? plan.region_bytes() * (size_t)d : 0);
        if (!own) RTR_CUDA_TRY(cudaMemsetAsync(st, 0, plan.region_bytes(), s));
        const int shift = lo + d * kRadixBits;
        if (plan.wide)
            k_radix_pass<unsigned long long><<<(unsigned)plan.tiles, kBlock, 0, s>>>(
                src, dst, n, shift, hist + d * kBins, (unsigned long long*)st, next + d, forms.wait_limit);
        else
            k_radix_pass<uint32_t><<<(unsigned)plan.tiles, kBlock, 0, s>>>(src, dst, n, shift, hist + d * kBins,
                                                                           (uint32_t*)st, next + d, forms.wait_limit);
        std::swap(src, dst);
    }
    t_launches += 1 + digits;
    RTR_CUDA_TRY(cudaGetLastError());
    *sorted = src;
    return RTR_OK;
}

int grid_for(int64_t work, int block, int blocks_per_sm)
{
    static const int sms = [] {  // initialised once, thread-safe
        int dev = 0, count = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || count <= 0)
            count = 148;
        return count;
    }();
    const int64_t need = (work + block - 1) / block;
    const int64_t cap = (int64_t)sms * blocks_per_sm;
    int64_t g = std::min<int64_t>(need, cap);
    return (int)std::max<int64_t>(1, g);
}

}  // namespace rtr
