// Weighted triangle counting, bit-exact to commonNbr
// (RTRex_Sequential/Escape/Decomposition.h:42-117).
//
// commonNbr finds every triangle once, in lexicographic order of its sorted
// vertex triple, and adds w = 1/double(du*dv*dw) to six directed-edge cells and
// three vertex cells.  Because of that discovery order:
//   perEdge[(x,y)]  = left fold, over common neighbours z of x and y in
//                     ascending z, of w(x,y,z)
//   perVertex[x]    = left fold over y in N(x) ascending, then over
//                     z in N(x) & N(y) with z > y ascending, of w(x,y,z)
// So each cell is produced by one thread as an ordered fold, with no
// floating-point atomics (the CUDA port's nine atomicAdd(double) per triangle,
// gpu_triangle_count.cu:70-88, give run-dependent bits).
//
// Kernels:
//   k_edge_fold    one thread per undirected edge: merge / galloping intersection
//                  of the two rows -> perEdge fold, live support, triangles with z>v
//   k_tri_fill     same intersection, writes the edge's triangle list
//                  {z, fwd(a,z), fwd(b,z), deg z} (used by the clean and for perVertex)
//   k_vertex_fold_light / _heavy  perVertex fold from the triangle lists: a thread
//                  per light vertex, a warp per heavy one
//   k_edge_count_heavy / k_tri_fill_heavy / k_pe_fold_heavy  the same for edges
//                  with deg u + deg v >= g->tune_edge, one warp per edge
// On large graphs (2m >= 2^25, or the rows layout forced) the rows of at least
// 256 entries get hash sets first (rowsets.cuh); an intersection whose longer
// row has one walks the shorter row against it (a warp per heavy edge four
// chunks of 32 per step, the heavy edges in the order of the sets they probe,
// so that the probed sets stay in L2); with at most 2^20 vertices, against a row
// of bits in shared memory where many edges share it (k_edge_count_bits).  The
// same pass also counts, for both
// slots of every edge, the common neighbours above the slot's neighbour (the
// rows layout's per-slot term counts, count_rows.cu), folds the heavy edges'
// perEdge in z order, and records each heavy edge's per-chunk hit masks for the
// rows layout's list fill.
// Three work-split parameters (g->tune_gallop: the row-length ratio above which
// an intersection gallops instead of merging; g->tune_heavy: the degree from
// which a vertex is folded by a warp; g->tune_edge: the degree sum from which an
// edge is intersected by a warp) change how work is spread, never a result; the
// autotuner (rtr_autotune) times candidates on the graph itself.
#include "fold_run.cuh"
#include "intersect.cuh"
#include "primitives.cuh"
#include "rowsets.cuh"
#include "rtr_graph.cuh"

#include <algorithm>
#include <memory>

namespace rtr {

namespace {

constexpr int kBlock = 256;

__device__ __forceinline__ void block_add_u64(unsigned long long v, unsigned long long* dst)
{
    __shared__ unsigned long long s[kBlock / 32];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) s[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long t = 0;
        for (int k = 0; k < kBlock / 32; ++k) t += s[k];
        if (t) atomicAdd(dst, t);
    }
}

// cgt (may be null): for each directed slot (x,y), the number of common
// neighbours z > y -- the terms slot (x,y) adds to perVertex[x] -- written for
// both slots of every edge (the rows layout's list offsets).
__global__ void __launch_bounds__(kBlock)
    k_edge_fold(const int64_t* __restrict__ off, const int32_t* __restrict__ nb, const int32_t* __restrict__ esrc,
                const int32_t* __restrict__ deg, const int32_t* __restrict__ fwd,
                const int32_t* __restrict__ partner, int64_t m, RowSets rs, double* __restrict__ pe,
                uint32_t* __restrict__ sup, int64_t* __restrict__ cnt, int64_t* __restrict__ cgt,
                unsigned long long* __restrict__ total, int gallop, int heavy_edge, int32_t* __restrict__ heavy_list,
                unsigned* __restrict__ nheavy)
{
    unsigned long long tri = 0;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = fwd[k];
        const int32_t u = esrc[i], v = nb[i];
        if (deg[u] + deg[v] >= heavy_edge) {  // a warp takes it (k_edge_count_heavy)
            if (heavy_list) heavy_list[atomicAdd(nheavy, 1u)] = (int32_t)k;
            continue;
        }
        const int64_t duv = (int64_t)deg[u] * (int64_t)deg[v];
        double acc = 0.0;
        uint32_t c = 0, above = 0, above_u = 0;
        thread_common(rs, off, nb, u, v, INT32_MIN, gallop, [&](int32_t z) {
            acc += 1.0 / (double)(duv * (int64_t)deg[z]);
            ++c;
            above += (z > v) ? 1u : 0u;
            above_u += (z > u) ? 1u : 0u;
        });
        pe[i] = acc;
        sup[i] = c;
        cnt[i] = c;
        if (cgt) {
            cgt[i] = above;
            cgt[partner[i]] = above_u;
        }
        tri += above;
    }
    block_add_u64(tri, total);
}

__global__ void __launch_bounds__(kBlock)
    k_tri_fill(const int64_t* __restrict__ off, const int32_t* __restrict__ nb, const int32_t* __restrict__ esrc,
               const int32_t* __restrict__ deg, const int32_t* __restrict__ partner, const int32_t* __restrict__ fwd,
               const int32_t* __restrict__ frank, int64_t m, const int64_t* __restrict__ tl_off,
               TriEntry* __restrict__ tl, int gallop, int heavy_edge)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = fwd[k];
        const int32_t u = esrc[i], v = nb[i];
        if (deg[u] + deg[v] >= heavy_edge) continue;  // k_tri_fill_heavy
        const int64_t duv = (int64_t)deg[u] * (int64_t)deg[v];
        int64_t w = tl_off[i];
        intersect_rows(nb, off[u], off[u + 1], off[v], off[v + 1], gallop, [&](int32_t z, int64_t pu, int64_t pv) {
            TriEntry t;
            t.z = z;
            t.eaz = (u < z) ? (int32_t)pu : partner[pu];
            t.ebz = (v < z) ? (int32_t)pv : partner[pv];
            t.dz = deg[z];
            t.wgt = 1.0 / (double)(duv * (int64_t)t.dz);
            t.raz = frank[t.eaz];
            t.rbz = frank[t.ebz];
            tl[w++] = t;
        });
    }
}

// Heavy edges (deg u + deg v >= heavy_edge), one warp each, dealt from the list
// the light edge fold built.  Counting is integer and order-free, so the lanes
// split the intersection (warp_intersect_part) and sum; the triangle list is
// written by the same split, each lane at its prefix offset, which keeps the
// entries in ascending z; perEdge is then folded from the list in that order
// (the same left fold over z ascending as the thread path).
constexpr int kHeavyEdgeBlock = 128;

// Lists layout: the count leaves, for the first m / 2 + 1 heavy edges, the hits
// before each lane's part of the intersection, so that k_tri_fill_heavy need not
// intersect twice (R-MAT, 500,000 edges: 1.43 -> 0.92 ms); 64 bytes an edge, in 16
// bits, so edges of more triangles than kPartsMax are intersected twice all the same.
constexpr int64_t kPartsMax = 65535;
// Edges from which the host learns the number of heavy ones first (15 us) and
// allocates no more than they need: half of 926,000 edges' notes were 30 MB that a
// graph of 2,500 heavy edges left unused, and made the pool map new memory now and
// then (a new graph's pass 22 ms, but up to 50).
constexpr int64_t kListFirst = 1ll << 18;
// Lists (with the clean's records) of up to this size may take the pool's cached
// blocks without leaving a margin to others.
constexpr double kListsSmall = 256.0 * (1ll << 20);

struct HeavyArgs {
    const int64_t* off;
    const int32_t* nb;
    const int32_t* esrc;
    const int32_t* deg;
    const int32_t* fwd;
    const int32_t* partner;
    const int32_t* heavy_list;
    int gallop;
    RowSets rs;
    uint32_t* sup;
    int64_t* cnt;
    int64_t* cgt;  // may be null; as in k_edge_fold
    double* pe;    // may be null: also fold perEdge of the heavy edges, in ascending z, from an ordered walk of
                   // the shorter row (the lists layout folds them from the lists instead, k_pe_fold_heavy)
    unsigned long long* total;
    const int64_t* moff;  // hit masks, for the rows layout's list fill (may be null)
    uint32_t* masks;
    uint16_t* parts;  // for k_tri_fill_heavy (kPartsMax)
    int64_t nparts;
};

// Heavy edges in the order of their longer row w (k_heavy_keys): a run is the
// edges of one w, apart for the priority rows' edges.  With at most 2^20 vertices
// a run that walks at least kRunWords words of 32 elements is cut into pieces of
// kPieceWords words, for k_edge_count_bits; the others are k_edge_count_heavy's.
// A piece sets up a row of at most 128 KB in a microsecond or two: 256 words (8,192
// bit tests) repay that, and pieces of 2,048 / 4,096 / 8,192 / 16,384 words take
// 39.4 / 38.8 / 38.8 / 38.3 ms for the count of R-MAT scale 19 and 108 / 100 / 96 /
// 94 for scale 20.  More vertices than fit one block's shared memory keep the hash
// sets: bits shared by several ids, with the hits looked up, took three times as
// long (scale 22: 950 ms for the heavy edges against 332).
// Heavy edges from which this pays, and from which the longest rows go ahead of the
// rest (count_rows.cu): each costs a few launches and waits.  R-MAT scales 15 / 16 /
// 17 / 18 (168,000 / 338,000 / 1.1 M / 2.2 M heavy edges), whole count: neither 4.48 /
// 6.81 / 13.5 / 27.6 ms, bits alone 5.02 / 6.72 / 12.4 / 24.1, both 5.33 / 6.72 / 11.4 /
// 18.7.
constexpr unsigned kBitsEdges = 1u << 18;
constexpr unsigned kAheadRows = 1u << 19;
constexpr int64_t kRunWords = 256;
constexpr int64_t kPieceWords = 8192;
constexpr int kMaxBits = 20;  // of the shared-memory row: 128 KB, a block an SM; below, two blocks
constexpr int kBitsBlock = 512, kBitsWide = 768;

struct HeavyRuns {
    const uint64_t* keys;  // per list place: w below wbits, the not-priority bit at wbits
    int wbits;
    int64_t n;
    const int64_t* poff;  // [2n + 1] first piece of run w (priority edges), n + w (others); null: no pieces
    const int32_t* fstart;  // [n] first slot of each vertex's neighbours above it

    __device__ __forceinline__ int64_t run(int64_t h) const
    {
        const uint32_t k = (uint32_t)keys[h];
        return (int64_t)(k & ((1u << wbits) - 1u)) + ((k >> wbits) & 1u ? n : 0);
    }
};

// One edge's walk, a warp's: the sums, and the hits not yet in the perEdge chain.
struct HeavyEdge {
    int32_t u, v;
    int64_t duv;
    int64_t mw0, mwn, word;  // the edge's mask words, and the next one
    unsigned c = 0, above = 0, above_u = 0;
    int pending = 0;
    double acc = 0.0;
};

struct alignas(16) HitBuf {
    int32_t z[160];  // 31 left over and a step's 128
    double w[32];
};

// The first cnt (<= 32) buffered hits enter the chain, in order.
__device__ __forceinline__ void chain_hits(const int32_t* __restrict__ deg, int64_t duv, HitBuf& hb, int base, int cnt,
                                           int lane, double& acc)
{
    hb.w[lane] = lane < cnt ? 1.0 / (double)(duv * (int64_t)deg[hb.z[base + lane]]) : 0.0;
    __syncwarp();
    const double2* w2 = reinterpret_cast<const double2*>(hb.w);
    if (cnt == 32) {
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const double2 x = w2[q];
            acc += x.x;
            acc += x.y;
        }
    } else {
        for (int q = 0; q < cnt; q += 2) {  // a missing weight is +0.0, which changes no sum that is not -0.0
            const double2 x = w2[q >> 1];
            acc += x.x;
            acc += x.y;
        }
    }
    __syncwarp();
}

// A step of B chunks of 32 elements of the shorter row, in ascending order.
template <int B>
__device__ __forceinline__ void take_step(const HeavyArgs& a, HeavyEdge& e, HitBuf& hb, const bool (&hit)[B],
                                          const int32_t (&x)[B], int lane)
{
    const unsigned lt = (1u << lane) - 1u;
    unsigned mine = 0;
    int tot = e.pending;
#pragma unroll
    for (int b = 0; b < B; ++b) {
        e.c += hit[b] ? 1u : 0u;
        e.above += (hit[b] && x[b] > e.v) ? 1u : 0u;
        e.above_u += (hit[b] && x[b] > e.u) ? 1u : 0u;
        const unsigned mb = __ballot_sync(0xffffffffu, hit[b]);
        if (lane == b) mine = mb;
        if (a.pe && hit[b]) hb.z[tot + __popc(mb & lt)] = x[b];
        tot += __popc(mb);
    }
    if (lane < B && e.word + lane < e.mwn) a.masks[e.mw0 + e.word + lane] = mine;
    e.word += B;
    if (!a.pe) return;
    if (tot >= 32) {
        __syncwarp();
        int done = 0;
        for (; tot - done >= 32; done += 32) chain_hits(a.deg, e.duv, hb, done, 32, lane, e.acc);
        tot -= done;
        const int32_t z = lane < tot ? hb.z[done + lane] : 0;
        __syncwarp();
        if (lane < tot) hb.z[lane] = z;
    }
    e.pending = tot;
}

__device__ __forceinline__ void finish_edge(const HeavyArgs& a, HeavyEdge& e, HitBuf& hb, int64_t i, int lane,
                                            unsigned long long& tri)
{
    if (a.pe && e.pending) {
        __syncwarp();
        chain_hits(a.deg, e.duv, hb, 0, e.pending, lane, e.acc);
    }
    e.c = __reduce_add_sync(0xffffffffu, e.c);
    e.above = __reduce_add_sync(0xffffffffu, e.above);
    e.above_u = __reduce_add_sync(0xffffffffu, e.above_u);
    if (lane == 0) {
        if (a.pe) a.pe[i] = e.acc;
        a.sup[i] = e.c;
        a.cnt[i] = e.c;
        if (a.cgt) {
            a.cgt[i] = e.above;
            a.cgt[a.partner[i]] = e.above_u;
        }
        tri += e.above;
    }
}

// The heavy edges [h0, h1) (h1 < 0: to the end) that no piece covers, a warp each.
__global__ void __launch_bounds__(kHeavyEdgeBlock, 6)
    k_edge_count_heavy(HeavyArgs a, HeavyRuns runs, int64_t h0, int64_t h1, const unsigned* __restrict__ nheavy,
                       unsigned long long* __restrict__ next)
{
    __shared__ HitBuf s_hits[kHeavyEdgeBlock / 32];
    const int lane = threadIdx.x & 31;
    HitBuf& hb = s_hits[threadIdx.x >> 5];
    const int64_t nh = h1 >= 0 ? h1 : (int64_t)*nheavy;
    const int64_t take = heavy_take(nh - h0);
    unsigned long long tri = 0;
    int64_t h = 0, hend = 0;
    while (true) {
        if (h >= hend && !next_heavy(next, h0, nh, take, h, hend)) break;
        const int64_t hh = h++;
        if (runs.poff) {
            const int64_t r = runs.run(hh);
            if (runs.poff[r + 1] > runs.poff[r]) continue;
        }
        const int64_t i = a.fwd[a.heavy_list[hh]];
        HeavyEdge e;
        e.u = a.esrc[i];
        e.v = a.nb[i];
        e.duv = (int64_t)a.deg[e.u] * (int64_t)a.deg[e.v];
        e.mw0 = a.masks ? a.moff[hh] : 0;
        e.mwn = a.masks ? a.moff[hh + 1] - e.mw0 : 0;
        e.word = 0;
        const int64_t u0 = a.off[e.u], u1 = a.off[e.u + 1], v0 = a.off[e.v], v1 = a.off[e.v + 1];
        // the shorter row walked against the longer one
        const bool u_short = u1 - u0 <= v1 - v0;
        const int32_t t = rs_table(a.rs, u_short ? e.v : e.u);
        if (t >= 0) {
            // 4 chunks per step, their lookups in flight together
            constexpr int B = 4;
            warp_probe_walk<B>(a.rs, t, a.nb, u_short ? u0 : v0, u_short ? u1 : v1, a.nb[(u_short ? v1 : u1) - 1],
                               lane, [&](const bool (&hit)[B], const int32_t (&x)[B]) {
                                   take_step<B>(a, e, hb, hit, x, lane);
                               });
        } else if (a.pe) {
            warp_walk(a.rs, a.off, a.nb, u_short ? u0 : v0, u_short ? u1 : v1, u_short ? e.v : e.u,
                      u_short ? v0 : u0, u_short ? v1 : u1, lane, [&](bool hit, int32_t z) {
                          const bool h1[1] = {hit};
                          const int32_t x1[1] = {z};
                          take_step<1>(a, e, hb, h1, x1, lane);
                      });
        } else {
            warp_intersect_part(a.nb, u0, u1, v0, v1, a.gallop, lane, [&](int32_t z, int64_t, int64_t) {
                ++e.c;
                e.above += (z > e.v) ? 1u : 0u;
                e.above_u += (z > e.u) ? 1u : 0u;
            });
            if (hh < a.nparts) {
                unsigned incl = e.c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += y;
                }
                a.parts[hh * 32 + lane] = (uint16_t)(incl - e.c);  // read only when the sum fits
            }
        }
        finish_edge(a, e, hb, i, lane, tri);
    }
    if (lane == 0 && tri) atomicAdd(a.total, tri);
}

// Pieces of long runs (n <= 2^lb): a block sets the row of w as bits in shared
// memory, and its warps walk the shorter rows against them, a bit test per
// element.  Against the hash sets (two 16-byte loads of a random bucket each) the
// walk was bound by the L1's lookups (95% of its peak at R-MAT scale 18); this one
// by instructions.  The hits below v and u (cgt) are counted in the one step that
// holds their places in the row.  Heavy edges of R-MAT scale 19 (4.7 M edges, 2.5 G
// tests): 23.4 -> 10.7 ms; scale 20: 56 -> 32.
__global__ void __launch_bounds__(1024, 1)
    k_edge_count_bits(HeavyArgs a, HeavyRuns runs, const longlong2* __restrict__ pieces, int64_t np, int lb,
                      unsigned long long* __restrict__ next)
{
    extern __shared__ __align__(16) unsigned char bits_raw[];
    unsigned* bm = reinterpret_cast<unsigned*>(bits_raw);
    HitBuf& hb = reinterpret_cast<HitBuf*>(bits_raw + ((size_t)1 << lb) / 8)[threadIdx.x >> 5];
    __shared__ long long s_piece;
    __shared__ int s_next;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    constexpr int B = 4;
    unsigned long long tri = 0;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) {
            s_piece = (long long)atomicAdd(next, 1ull);
            s_next = 0;
        }
        __syncthreads();
        if (s_piece >= np) break;
        const longlong2 pc = pieces[s_piece];
        if (pc.x >= pc.y) continue;
        uint4* b4 = reinterpret_cast<uint4*>(bm);
        for (int k = threadIdx.x; k < (1 << lb) / 128; k += blockDim.x) b4[k] = make_uint4(0, 0, 0, 0);
        const int32_t w = (int32_t)(runs.run(pc.x) % runs.n);
        const int64_t w0 = a.off[w], w1 = a.off[w + 1];
        const int32_t dw = a.deg[w];
        __syncthreads();
        for (int64_t j = w0 + threadIdx.x; j < w1; j += blockDim.x) {
            const uint32_t x = (uint32_t)a.nb[j];
            atomicOr(&bm[x >> 5], 1u << (x & 31));
        }
        __syncthreads();
        // up to 8 edges at a time, so that every warp takes several times
        const int64_t share = (pc.y - pc.x) / (int64_t)(blockDim.x / 32 * 8);
        const int take = share < 1 ? 1 : share < 8 ? (int)share : 8;
        while (true) {
            int k0 = 0;
            if (lane == 0) k0 = atomicAdd(&s_next, take);
            const int64_t h0 = pc.x + __shfl_sync(0xffffffffu, k0, 0);
            if (h0 >= pc.y) break;
            const int ne = pc.y - h0 < take ? (int)(pc.y - h0) : take;
            // the take's edges, one per lane
            int32_t ei = 0, er = 0, es0 = 0, elen = 0, edy = 0, epv = 0, epu = 0;
            int64_t em = 0;
            if (lane <= ne && a.masks) em = a.moff[h0 + lane];
            if (lane < ne) {
                ei = a.fwd[a.heavy_list[h0 + lane]];
                er = a.partner[ei];
                const int32_t u = a.esrc[ei], v = a.nb[ei];
                const int32_t y = u == w ? v : u;
                es0 = (int32_t)a.off[y];
                elen = (int32_t)(a.off[y + 1] - es0);
                edy = a.deg[y];
                const int32_t past_w = (y == u ? ei : er) - es0 + 1, past_y = runs.fstart[y] - es0;
                epv = y == u ? past_w : past_y;
                epu = y == u ? past_y : past_w;
            }
            for (int k = 0; k < ne; ++k) {
                const int32_t* row = a.nb + __shfl_sync(0xffffffffu, es0, k);
                const int len = __shfl_sync(0xffffffffu, elen, k);
                const int pv = __shfl_sync(0xffffffffu, epv, k), pu = __shfl_sync(0xffffffffu, epu, k);
                const int64_t duv = (int64_t)dw * (int64_t)__shfl_sync(0xffffffffu, edy, k);
                const int64_t mw0 = __shfl_sync(0xffffffffu, em, k);
                const int mwn = (int)(__shfl_sync(0xffffffffu, em, k + 1) - mw0);
                int c = 0, below_v = -1, below_u = -1, pending = 0;
                double acc = 0.0;
                uint32_t xn[B];  // past the end: w, which is not in its own row
#pragma unroll
                for (int b = 0; b < B; ++b) xn[b] = 32 * b + lane < len ? row[32 * b + lane] : w;
                for (int base = 0; base < len; base += 32 * B) {
                    uint32_t x[B];
                    unsigned mb[B], mine = 0;
                    bool hit[B];
#pragma unroll
                    for (int b = 0; b < B; ++b) {
                        x[b] = xn[b];
                        const int p = base + 32 * (B + b) + lane;
                        xn[b] = p < len ? row[p] : w;
                    }
#pragma unroll
                    for (int b = 0; b < B; ++b) {
                        hit[b] = (bm[x[b] >> 5] >> (x[b] & 31)) & 1u;
                        mb[b] = __ballot_sync(0xffffffffu, hit[b]);
                        if (lane == b) mine = mb[b];
                    }
                    int tot = pending;
#pragma unroll
                    for (int b = 0; b < B; ++b) {
                        if (hit[b]) hb.z[tot + __popc(mb[b] & lt)] = (int32_t)x[b];
                        tot += __popc(mb[b]);
                    }
                    auto below = [&](int at) {  // hits before place `at` of the row, in this step or earlier
                        int r = c;
#pragma unroll
                        for (int b = 0; b < B; ++b) {
                            const int q = at - base - 32 * b;
                            r += q <= 0 ? 0 : __popc(q >= 32 ? mb[b] : mb[b] & ((1u << q) - 1u));
                        }
                        return r;
                    };
                    if ((unsigned)(pv - base) < 32u * B) below_v = below(pv);
                    if ((unsigned)(pu - base) < 32u * B) below_u = below(pu);
                    c += tot - pending;
                    if (lane < B && (base >> 5) + lane < mwn) a.masks[mw0 + (base >> 5) + lane] = mine;
                    if (tot >= 32) {
                        __syncwarp();
                        int done = 0;
                        for (; tot - done >= 32; done += 32) chain_hits(a.deg, duv, hb, done, 32, lane, acc);
                        tot -= done;
                        const int32_t z = lane < tot ? hb.z[done + lane] : 0;
                        __syncwarp();
                        if (lane < tot) hb.z[lane] = z;
                    }
                    pending = tot;
                }
                __syncwarp();
                if (pending) chain_hits(a.deg, duv, hb, 0, pending, lane, acc);
                const int64_t i = __shfl_sync(0xffffffffu, ei, k), r = __shfl_sync(0xffffffffu, er, k);
                if (lane == 0) {
                    const int above = below_v < 0 ? 0 : c - below_v;
                    a.pe[i] = acc;
                    a.sup[i] = (uint32_t)c;
                    a.cnt[i] = c;
                    a.cgt[i] = above;
                    a.cgt[r] = below_u < 0 ? 0 : c - below_u;
                    tri += (unsigned long long)above;
                }
            }
        }
    }
    if (lane == 0 && tri) atomicAdd(a.total, tri);
}

// The first slot of each vertex's neighbours above it.
__global__ void k_fwd_start(const int64_t* __restrict__ off, const int32_t* __restrict__ nb, int64_t n,
                            int32_t* __restrict__ fstart)
{
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        fstart[v] = (int32_t)lower_bound_row(nb, off[v], off[v + 1], (int32_t)v);
}

// First and last place of each run in the list.
__global__ void k_run_ends(HeavyRuns runs, int64_t nh, int32_t* __restrict__ first, int32_t* __restrict__ last)
{
    for (int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; h < nh; h += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = runs.run(h);
        if (h == 0 || runs.run(h - 1) != r) first[r] = (int32_t)h;
        if (h + 1 == nh || runs.run(h + 1) != r) last[r] = (int32_t)h + 1;
    }
}

// Pieces of each run (`pre`: the words of the list's edges, scanned).
__global__ void k_piece_counts(const int32_t* __restrict__ first, const int32_t* __restrict__ last,
                               const int64_t* __restrict__ pre, RowSets rs, int64_t n, int64_t* __restrict__ cnt)
{
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r <= 2 * n; r += (int64_t)gridDim.x * blockDim.x) {
        int64_t c = 0;
        if (r < 2 * n && last[r] > first[r] && rs_table(rs, (int32_t)(r % n)) >= 0) {
            const int64_t words = pre[last[r]] - pre[first[r]];
            if (words >= kRunWords) c = (words + kPieceWords - 1) / kPieceWords;
        }
        cnt[r] = c;
    }
}

// Piece j of a run: its edges whose words begin in [j, j + 1) x kPieceWords of the run's.
__global__ void k_pieces(const int32_t* __restrict__ first, const int32_t* __restrict__ last,
                         const int64_t* __restrict__ pre, const int64_t* __restrict__ poff, int64_t n, int64_t np,
                         longlong2* __restrict__ pieces)
{
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < np; p += (int64_t)gridDim.x * blockDim.x) {
        int64_t lo = 0, hi = 2 * n;  // the last run whose first piece is at most p
        while (hi - lo > 1) {
            const int64_t mid = (lo + hi) >> 1;
            if (poff[mid] <= p) lo = mid;
            else hi = mid;
        }
        const int64_t f = first[lo], l = last[lo], target = pre[f] + (p - poff[lo]) * kPieceWords;
        auto at = [&](int64_t t) {  // the first edge whose words begin at t or later
            int64_t x = f, y = l;
            while (x < y) {
                const int64_t mid = (x + y) >> 1;
                if (pre[mid] < t) x = mid + 1;
                else y = mid;
            }
            return x;
        };
        pieces[p] = make_longlong2(at(target), at(target + kPieceWords));
    }
}

// The heavy edges alone, where they are to be counted before the light ones.
__global__ void k_heavy_list(const int32_t* __restrict__ esrc, const int32_t* __restrict__ nb,
                             const int32_t* __restrict__ deg, const int32_t* __restrict__ fwd, int64_t m,
                             int heavy_edge, int32_t* __restrict__ heavy_list, unsigned* __restrict__ nheavy)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = fwd[k];
        if (deg[esrc[i]] + deg[nb[i]] >= heavy_edge) heavy_list[atomicAdd(nheavy, 1u)] = (int32_t)k;
    }
}

// Heavy edges keyed by the vertex whose hash set their intersection probes
// (the longer row; the shorter one is walked): sorted on it, the warps running
// at any one time probe a few sets, which then stay in L2.
__global__ void k_heavy_keys(const int64_t* __restrict__ off, const int32_t* __restrict__ esrc,
                             const int32_t* __restrict__ nb, const int32_t* __restrict__ fwd,
                             const int32_t* __restrict__ heavy_list, int64_t nh,
                             const int32_t* __restrict__ rank, int nbits, uint64_t* __restrict__ keys,
                             unsigned* __restrict__ npri)
{
    for (int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; h < nh; h += (int64_t)gridDim.x * blockDim.x) {
        const int32_t k = heavy_list[h];
        const int64_t i = fwd[k];
        const int32_t u = esrc[i], v = nb[i];
        const int32_t w = off[u + 1] - off[u] <= off[v + 1] - off[v] ? v : u;
        // edges of the priority rows first
        const bool pri = rank && (rank[u] >= 0 || rank[v] >= 0);
        if (pri) atomicAdd(npri, 1u);
        keys[h] = ((uint64_t)(uint32_t)k << 32) | ((uint64_t)(pri ? 0 : 1) << nbits) | (uint64_t)(uint32_t)w;
    }
}

// Hit-mask words of each heavy edge: one per 32 elements of its shorter row
// when the longer row has a hash set (the edges the count walks through one),
// else none.
__global__ void k_mask_words(const int64_t* __restrict__ off, const int32_t* __restrict__ esrc,
                             const int32_t* __restrict__ nb, const int32_t* __restrict__ fwd,
                             const int32_t* __restrict__ heavy_list, int64_t nh, RowSets rs,
                             int64_t* __restrict__ words)
{
    for (int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; h <= nh; h += (int64_t)gridDim.x * blockDim.x) {
        if (h == nh) {
            words[h] = 0;
            continue;
        }
        const int64_t i = fwd[heavy_list[h]];
        const int32_t u = esrc[i], v = nb[i];
        const int64_t du = off[u + 1] - off[u], dv = off[v + 1] - off[v];
        const bool u_short = du <= dv;
        words[h] = rs_table(rs, u_short ? v : u) >= 0 ? ((u_short ? du : dv) + 31) / 32 : 0;
    }
}

__global__ void k_heavy_order(const uint64_t* __restrict__ keys, int64_t nh, int32_t* __restrict__ heavy_list)
{
    for (int64_t h = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; h < nh; h += (int64_t)gridDim.x * blockDim.x)
        heavy_list[h] = (int32_t)(keys[h] >> 32);
}

__global__ void __launch_bounds__(kHeavyEdgeBlock)
    k_tri_fill_heavy(const int64_t* __restrict__ off, const int32_t* __restrict__ nb, const int32_t* __restrict__ esrc,
                     const int32_t* __restrict__ deg, const int32_t* __restrict__ partner,
                     const int32_t* __restrict__ fwd, const int32_t* __restrict__ frank,
                     const int32_t* __restrict__ heavy_list, const unsigned* __restrict__ nheavy, int gallop,
                     const uint16_t* __restrict__ parts, int64_t nparts, const int64_t* __restrict__ tl_off,
                     TriEntry* __restrict__ tl, unsigned long long* __restrict__ next)
{
    const int lane = threadIdx.x & 31;
    const int64_t nh = *nheavy;
    const int64_t take = heavy_take(nh);
    int64_t hq = 0, hend = 0;
    while (true) {
        if (hq >= hend && !next_heavy(next, 0, nh, take, hq, hend)) break;
        const int64_t h = hq++;
        const int64_t i = fwd[heavy_list[h]];
        const int32_t u = esrc[i], v = nb[i];
        const int64_t duv = (int64_t)deg[u] * (int64_t)deg[v];
        int64_t w = tl_off[i];
        if (h < nparts && tl_off[i + 1] - w <= kPartsMax) {
            w += parts[h * 32 + lane];
        } else {
            unsigned c = 0;
            warp_intersect_part(nb, off[u], off[u + 1], off[v], off[v + 1], gallop, lane,
                                [&](int32_t, int64_t, int64_t) { ++c; });
            unsigned incl = c;  // inclusive prefix over lanes
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            w += incl - c;
        }
        warp_intersect_part(nb, off[u], off[u + 1], off[v], off[v + 1], gallop, lane,
                            [&](int32_t z, int64_t pu, int64_t pv) {
                                TriEntry t;
                                t.z = z;
                                t.eaz = (u < z) ? (int32_t)pu : partner[pu];
                                t.ebz = (v < z) ? (int32_t)pv : partner[pv];
                                t.dz = deg[z];
                                t.wgt = 1.0 / (double)(duv * (int64_t)t.dz);
                                t.raz = frank[t.eaz];
                                t.rbz = frank[t.ebz];
                                tl[w++] = t;
                            });
    }
}

__global__ void __launch_bounds__(kHeavyEdgeBlock)
    k_pe_fold_heavy(const int32_t* __restrict__ fwd, const int32_t* __restrict__ heavy_list,
                    const unsigned* __restrict__ nheavy, const int64_t* __restrict__ tl_off,
                    const TriEntry* __restrict__ tl, double* __restrict__ pe)
{
    __shared__ double s_w[kHeavyEdgeBlock / 32][32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t nh = *nheavy;
    const int64_t nwarps = (int64_t)gridDim.x * (kHeavyEdgeBlock / 32);
    for (int64_t h = (int64_t)blockIdx.x * (kHeavyEdgeBlock / 32) + wib; h < nh; h += nwarps) {
        const int64_t i = fwd[heavy_list[h]];
        const int64_t e0 = tl_off[i], e1 = tl_off[i + 1];
        double acc = 0.0;
        for (int64_t b = e0; b < e1; b += 32) {
            if (b + lane < e1) s_w[wib][lane] = tl[b + lane].wgt;
            __syncwarp();
            const int cnt = e1 - b < 32 ? (int)(e1 - b) : 32;
            for (int j = 0; j < cnt; ++j) acc += s_w[wib][j];
            __syncwarp();
        }
        if (lane == 0) pe[i] = acc;
    }
}

// perVertex[x] = left fold over y in N(x) ascending, then z > y ascending, of the
// triangle weights (Decomposition.h:95-101).  Slot i = (x,y) adds the last
// cgt[i] entries of its edge's list (those with z > y).  Bound by one dependent
// double add per term of the largest vertex (8 cycles each, 4.1 ns).
//
// k_fold_gather copies the terms' weights into fold order (lpos, the scan of
// cgt over the slots): eight lanes per slot.  Then a vertex's terms lie side by
// side: k_fold_terms_light folds a vertex of fewer than kFoldWarp terms per
// thread, k_fold_terms_heavy one of more per warp (fold_run.cuh).  Vertices are
// dealt by id modulo the warp count (power-law generators put hubs at
// neighbouring ids).
// [lo, hi): the degrees taken.  From kAheadEdges heavy edges on, the vertices whose
// edges are all heavy (those of tune_edge neighbours and more) are gathered and
// folded as soon as the heavy lists are there, on the second stream, all of them a
// warp each, beside the light lists and the other vertices: the longest chain, 0.79
// ms of R-MAT 500,009 edges, no longer runs alone at the end.  Count of that graph
// (162,000 heavy edges) 3.75 -> 3.12 ms, of 203,311 edges (30,000 heavy) 2.03 -> 1.69,
// of 40,000 (1,100 heavy) 0.05 ms less -- below the 0.1 ms that making the stream
// costs a new graph.
//   R-MAT, 500,009 edges, 6.1 M triangles, in one go: 5.58 -> 0.92 ms; 203,311 edges, 2.0 M
//   triangles: 3.37 -> 0.57 ms (before: a binary search per slot for its first
//   entry, and per 32 terms a search, a gather and the adds, none overlapped).
constexpr int kFoldWarp = 64;
constexpr unsigned kAheadEdges = 16384;
// The gather visits every slot: it pays from one term per this many slots on
// (4,152 terms over 10,000 slots 0.023 against 0.050 ms folded from the lists,
// 358,398 over 1.85 M 0.11 against 0.13; but 23,409 over 400,000 0.038 against 0.029).
constexpr int64_t kSlotsPerTerm = 8;

__global__ void __launch_bounds__(kBlock)
    k_fold_gather(const int32_t* __restrict__ esrc, const int32_t* __restrict__ nb, const int32_t* __restrict__ partner,
                  const int32_t* __restrict__ deg, int lo, int hi, int64_t m2, const int64_t* __restrict__ cgt,
                  const int64_t* __restrict__ lpos, const int64_t* __restrict__ tl_off,
                  const TriEntry* __restrict__ tl, double* __restrict__ terms)
{
    const int sub = threadIdx.x & 7;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3; i < m2;
         i += ((int64_t)gridDim.x * blockDim.x) >> 3) {
        const int64_t len = cgt[i];
        const int32_t x = esrc[i], d = deg[x];
        if (len == 0 || d < lo || d >= hi) continue;
        const int64_t c = x < nb[i] ? i : (int64_t)partner[i];
        const TriEntry* from = tl + (tl_off[c + 1] - len);
        double* to = terms + lpos[i];
        for (int64_t j = sub; j < len; j += 8) to[j] = from[j].wgt;
    }
}

__global__ void __launch_bounds__(kBlock)
    k_fold_terms_light(const int64_t* __restrict__ off, const int64_t* __restrict__ lpos, int64_t n, int hi,
                       const double* __restrict__ terms, double* __restrict__ pv)
{
    for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
        const int64_t p0 = lpos[off[x]], p1 = lpos[off[x + 1]];
        if (p1 - p0 >= kFoldWarp || off[x + 1] - off[x] >= hi) continue;
        double acc = 0.0;
        for (int64_t p = p0; p < p1; ++p) acc += terms[p];
        pv[x] = acc;
    }
}

constexpr int kHeavyBlock = 128;
__global__ void __launch_bounds__(kHeavyBlock)
    k_fold_terms_heavy(const int64_t* __restrict__ off, const int64_t* __restrict__ lpos, int64_t n, int lo, int hi,
                       const double* __restrict__ terms, double* __restrict__ pv)
{
    __shared__ __align__(16) double s_w[kHeavyBlock / 32][kFoldStep];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t nwarps = (int64_t)gridDim.x * (kHeavyBlock / 32);
    for (int64_t x = (int64_t)blockIdx.x * (kHeavyBlock / 32) + wib; x < n; x += nwarps) {
        const int64_t p0 = lpos[off[x]], p1 = lpos[off[x + 1]];
        const int64_t d = off[x + 1] - off[x];
        if ((p1 - p0 < kFoldWarp && lo == 0) || d < lo || d >= hi) continue;
        const double acc = fold_run<false>(terms + p0, p1 - p0, 0.0, s_w[wib]);
        if (lane == 0) pv[x] = acc;
    }
}

// The same fold straight from the lists, without the terms' array: for graphs of
// few triangles (fewer launches), or when there is no room for it.
//
// k_vertex_fold_light: one thread per vertex of degree < heavy (at most
// heavy^2/2 entries each).
__global__ void __launch_bounds__(kBlock)
    k_vertex_fold_light(const int64_t* __restrict__ off, const int32_t* __restrict__ nb,
                        const int32_t* __restrict__ deg, const int32_t* __restrict__ partner, int64_t n,
                        const int64_t* __restrict__ cgt, const int64_t* __restrict__ tl_off,
                        const TriEntry* __restrict__ tl, double* __restrict__ pv, int heavy)
{
    for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
        if (deg[x] >= heavy) continue;
        double acc = 0.0;
        for (int64_t i = off[x]; i < off[x + 1]; ++i) {
            const int64_t len = cgt[i];
            if (len == 0) continue;
            const int64_t c = (x < nb[i]) ? i : (int64_t)partner[i];
            const int64_t hi = tl_off[c + 1];
            for (int64_t p = hi - len; p < hi; ++p) acc += tl[p].wgt;
        }
        pv[x] = acc;
    }
}

// k_vertex_fold_heavy: one warp per vertex of degree >= heavy, dealt by id
// modulo the warp count.  Per 32 neighbours the lanes find their entry ranges at
// once; the ranges' entries are then loaded 32 at a time in fold order (each lane
// finds its range by a 5-step search over the range ends in shared memory),
// staged in shared memory, and added in order.
__global__ void __launch_bounds__(kHeavyBlock)
    k_vertex_fold_heavy(const int64_t* __restrict__ off, const int32_t* __restrict__ nb,
                        const int32_t* __restrict__ deg, const int32_t* __restrict__ partner, int64_t n,
                        const int64_t* __restrict__ cgt, const int64_t* __restrict__ tl_off,
                        const TriEntry* __restrict__ tl, double* __restrict__ pv, int heavy)
{
    __shared__ int64_t s_end[kHeavyBlock / 32][32];
    __shared__ int64_t s_beg[kHeavyBlock / 32][32];
    __shared__ double s_w[kHeavyBlock / 32][32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t nwarps = (int64_t)gridDim.x * (kHeavyBlock / 32);
    for (int64_t hx = (int64_t)blockIdx.x * (kHeavyBlock / 32) + wib; hx < n; hx += nwarps) {
        if (deg[hx] < heavy) continue;  // uniform across the warp
        const int64_t h0 = off[hx], h1 = off[hx + 1];
        double acc = 0.0;
        for (int64_t cb = h0; cb < h1; cb += 32) {
            const int64_t i = cb + lane;
            int64_t a = 0, len = 0;
            if (i < h1) {
                len = cgt[i];
                const int64_t c = (hx < nb[i]) ? i : (int64_t)partner[i];
                a = tl_off[c + 1] - len;
            }
            int64_t end = len;  // inclusive prefix of the range lengths
            for (int o = 1; o < 32; o <<= 1) {
                const int64_t t = __shfl_up_sync(0xffffffffu, end, o);
                if (lane >= o) end += t;
            }
            s_end[wib][lane] = end;
            s_beg[wib][lane] = a - (end - len);  // entry index = s_beg[owner] + k
            __syncwarp();
            const int64_t total = s_end[wib][31];
            for (int64_t k0 = 0; k0 < total; k0 += 32) {
                const int64_t k = k0 + lane;
                if (k < total) {
                    int lo = 0, hi = 31;  // first lane whose range ends after k
                    while (lo < hi) {
                        const int mid = (lo + hi) >> 1;
                        if (s_end[wib][mid] <= k) lo = mid + 1;
                        else hi = mid;
                    }
                    s_w[wib][lane] = tl[s_beg[wib][lo] + k].wgt;
                }
                __syncwarp();
                const int cnt = total - k0 < 32 ? (int)(total - k0) : 32;
                for (int j = 0; j < cnt; ++j) acc += s_w[wib][j];
                __syncwarp();
            }
            __syncwarp();  // the ranges are rewritten next
        }
        if (lane == 0) pv[hx] = acc;
    }
}

// The pieces of the list's long runs; none (runs->poff null) when there is no room.
int cut_runs(rtr_graph* g, Scratch& sc, const RowSets& rs, int64_t nh, const int64_t* pre, HeavyRuns* runs,
             longlong2** pieces, int64_t* np)
{
    cudaStream_t s = g->stream;
    const int64_t n = g->n;
    int32_t* ends = (int32_t*)sc.get(sizeof(int32_t) * 4 * (n + 1));
    int64_t* pcnt = (int64_t*)sc.get(sizeof(int64_t) * (2 * n + 1));
    int64_t* poff = (int64_t*)sc.get(sizeof(int64_t) * (2 * n + 1));
    int64_t* tmp = (int64_t*)sc.get(sizeof(int64_t) * scan_temp_elems(2 * n + 1));
    int32_t* fstart = (int32_t*)sc.get(sizeof(int32_t) * (n + 1));
    if (!ends || !pcnt || !poff || !tmp || !fstart) {
        cudaGetLastError();
        return RTR_OK;
    }
    int32_t *first = ends, *last = ends + 2 * (n + 1);
    RTR_CUDA_TRY(cudaMemsetAsync(ends, 0, sizeof(int32_t) * 4 * (n + 1), s));
    k_fwd_start<<<grid_for(n, 256), 256, 0, s>>>(g->offsets, g->nbors, n, fstart);
    k_run_ends<<<grid_for(nh, 256), 256, 0, s>>>(*runs, nh, first, last);
    k_piece_counts<<<grid_for(2 * n + 1, 256), 256, 0, s>>>(first, last, pre, rs, n, pcnt);
    RTR_TRY(exclusive_scan_i64(pcnt, poff, 2 * n + 1, nullptr, tmp, s));
    g->launches += 3 + take_primitive_launches();
    int64_t all = 0;
    if (const int rc = read_words(g, &np[0], poff + n, sizeof(int64_t))) return rc;
    if (const int rc = read_words(g, &all, poff + 2 * n, sizeof(int64_t))) return rc;
    np[1] = all - np[0];
    if (all == 0) return RTR_OK;
    *pieces = (longlong2*)sc.get(sizeof(longlong2) * (size_t)all);
    if (!*pieces) {
        cudaGetLastError();
        np[0] = np[1] = 0;
        return RTR_OK;
    }
    k_pieces<<<grid_for(all, 256), 256, 0, s>>>(first, last, pre, poff, n, all, *pieces);
    g->launches += 1;
    runs->poff = poff;
    runs->fstart = fstart;
    return RTR_OK;
}

int launch_bits(rtr_graph* g, const HeavyArgs& ha, const HeavyRuns& runs, const longlong2* pieces, int64_t np,
                unsigned long long* next)
{
    if (np == 0) return RTR_OK;
    const int nb = bits_for((uint64_t)(g->n > 1 ? g->n - 1 : 1));
    const int lb = nb < 10 ? 10 : nb < kMaxBits ? nb : kMaxBits;
    const int threads = lb == kMaxBits ? kBitsWide : kBitsBlock;
    const size_t smem = ((size_t)1 << lb) / 8 + sizeof(HitBuf) * (threads / 32);
    RTR_CUDA_TRY(cudaFuncSetAttribute(k_edge_count_bits, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int64_t grid = std::min<int64_t>(np, grid_for(1ll << 40, threads, lb == kMaxBits ? 1 : 2));
    k_edge_count_bits<<<(unsigned)grid, threads, smem, g->stream>>>(ha, runs, pieces, np, lb, next);
    g->launches += 1;
    RTR_CUDA_TRY(cudaGetLastError());
    return RTR_OK;
}

}  // namespace

int count_triangles(rtr_graph* g)
{
    take_primitive_launches();  // what a call that failed left uncounted is not this one's
    if (g->stage < 1) {
        set_error("count called before the graph was built");
        return RTR_ERR_STATE;
    }
    cudaStream_t s = g->stream;
    const int64_t n = g->n, m2 = g->m2, m = g->m;
    if (!g->pe) {
        g->pe = (double*)dev_alloc(g, sizeof(double) * (m2 + 1));
        g->pv = (double*)dev_alloc(g, sizeof(double) * (n + 1));
        g->sup = (uint32_t*)dev_alloc(g, sizeof(uint32_t) * (m2 + 1));
        g->st = (uint8_t*)dev_alloc(g, m2 + 16);
        g->tl_off = (int64_t*)dev_alloc(g, sizeof(int64_t) * (m2 + 1));
        if (!g->pe || !g->pv || !g->sup || !g->st || !g->tl_off) {
            set_error("device allocation failed for the triangle state");
            return RTR_ERR_CUDA;
        }
    }
    Scratch sc(g);
    int64_t* cnt = (int64_t*)sc.get(sizeof(int64_t) * (m2 + 1));
    int64_t* tmp = (int64_t*)sc.get(sizeof(int64_t) * scan_temp_elems(m2 + 1));
    int32_t* heavy_list = (int32_t*)sc.get(sizeof(int32_t) * (m + 1));
    unsigned* nheavy = (unsigned*)(g->ctr + 5);  // heavy edges; those of the priority rows
    // a queue word for each launch that deals the heavy edges: the counts', then the list fill's
    constexpr int kQueues = 6;
    unsigned long long* hq = (unsigned long long*)sc.get(sizeof(unsigned long long) * kQueues);
    if (!cnt || !tmp || !heavy_list || !hq) {
        set_error("device allocation failed (count scratch)");
        return RTR_ERR_CUDA;
    }
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    RTR_CUDA_TRY(cudaMemsetAsync(g->ctr, 0, 8 * sizeof(unsigned long long), s));
    RTR_CUDA_TRY(cudaMemsetAsync(cnt, 0, sizeof(int64_t) * (m2 + 1), s));
    RTR_CUDA_TRY(cudaMemsetAsync(g->pe, 0, sizeof(double) * (m2 + 1), s));
    RTR_CUDA_TRY(cudaMemsetAsync(g->sup, 0, sizeof(uint32_t) * (m2 + 1), s));
    const int ge = grid_for(m, kBlock);
    const int gh = grid_for(1ll << 40, kHeavyEdgeBlock, 16);
    const int gc = grid_for(1ll << 40, kHeavyEdgeBlock, 6);  // k_edge_count_heavy: the resident blocks
    RTR_CUDA_TRY(cudaMemsetAsync(hq, 0, sizeof(unsigned long long) * kQueues, s));
    ktime_begin(g, KT_EDGE_FOLD);
    // Hash sets of the long rows, for the heavy-edge count and the rows layout:
    // built when the rows layout is asked for, or may be chosen (2m >= count_sets).
    RowSets rs{nullptr, nullptr, nullptr, nullptr};
    if (g->count_mode == 2 || (g->count_mode == 0 && m2 >= g->count_sets)) {
        const int rc = build_row_sets(g, sc, kSetDegree, &rs);
        if (rc) return rc;
    }
    // per-slot counts of perVertex terms
    int64_t* cgt = (int64_t*)sc.get(sizeof(int64_t) * (m2 + 1));
    if (!cgt) {
        set_error("device allocation failed (count scratch)");
        return RTR_ERR_CUDA;
    }
    RTR_CUDA_TRY(cudaMemsetAsync(cgt, 0, sizeof(int64_t) * (m2 + 1), s));
    // heavy-edge perEdge folded by the count when the rows layout is likely
    const bool heavy_pe = g->count_mode == 2 || rs.tab != nullptr;
    // The light edges, and the list of the heavy ones; with the rows layout likely, the light edges
    // wait until the longest perVertex chains (below) are under way.
    auto light = [&](int32_t* list) {
        ktime_begin(g, KT_EDGE_LIGHT);
        k_edge_fold<<<ge, kBlock, 0, s>>>(g->offsets, g->nbors, g->esrc, g->deg, g->fwd, g->partner, m, rs, g->pe,
                                          g->sup, cnt, cgt, g->ctr, g->tune_gallop, g->tune_edge, list, nheavy);
        ktime_end(g, KT_EDGE_LIGHT);
    };
    int64_t nparts = 0;  // heavy edges noted for k_tri_fill_heavy
    if (rs.tab || (!heavy_pe && m >= kListFirst)) {
        k_heavy_list<<<ge, kBlock, 0, s>>>(g->esrc, g->nbors, g->deg, g->fwd, m, g->tune_edge, heavy_list, nheavy);
        g->launches += 1;
    } else {
        light(heavy_list);
    }
    if (!rs.tab && !heavy_pe) {
        nparts = m / 2 + 1;
        if (m >= kListFirst) {
            unsigned nh = 0;
            if (const int rc = read_words(g, &nh, nheavy, sizeof nh)) return rc;
            nparts = std::min<int64_t>(nparts, nh);
            light(nullptr);
        }
    }
    // the longest perVertex chains ahead of the rest, where the rows layout is likely.  Not when this
    // graph holds lists from an earlier count (they will be kept again), nor under a set window size
    // (the caller's bound is then on all the lists that are held).
    PriorityRows pr;
    unsigned nh = 0;  // heavy edges, where the sets are built
    if (rs.tab)
        if (const int rc = read_words(g, &nh, nheavy, sizeof(unsigned))) return rc;
    if (rs.tab && !g->tl && g->rows_window_cap == 0 && nh >= kAheadRows) {
        const int rc = pick_priority_rows(g, sc, &pr);
        if (rc) return rc;
    }
    if (pr.count == 0) release_owned(g, &g->rows_ahead, &g->rows_ahead_cap);
    struct SideGuard {  // the second stream is done with the scratch before it is released
        rtr_graph* g;
        PriorityRows* pr;
        cudaEvent_t lists = nullptr;
        ~SideGuard()
        {
            if ((pr->folding || lists) && g->side) cudaStreamSynchronize(g->side);
            if (lists) cudaEventDestroy(lists);
            if (pr->begin) cudaEventDestroy(pr->begin);
            if (pr->end) cudaEventDestroy(pr->end);
        }
    } side_guard{g, &pr};
    HeavyRuns runs{nullptr, 0, n, nullptr, nullptr};
    if (rs.tab) {  // heavy edges in the order of the sets they probe
        if (nh > 1) {
            uint64_t* hkeys = (uint64_t*)sc.get(sizeof(uint64_t) * (nh + 1));
            uint64_t* halt = (uint64_t*)sc.get(sizeof(uint64_t) * (nh + 1));
            void* htmp = sc.get(radix_temp_bytes(nh));
            if (!hkeys || !halt || !htmp) {
                set_error("device allocation failed (heavy-edge order)");
                return RTR_ERR_CUDA;
            }
            const int nbits = bits_for((uint64_t)(n > 0 ? n - 1 : 0));
            k_heavy_keys<<<grid_for(nh, 256), 256, 0, s>>>(g->offsets, g->esrc, g->nbors, g->fwd, heavy_list, nh,
                                                            pr.rank, nbits, hkeys, nheavy + 1);
            uint64_t* sorted = nullptr;
            RTR_TRY(radix_sort_u64(hkeys, halt, nh, nbits + (pr.count > 0 ? 1 : 0), htmp, s, &sorted));
            unsigned npri = 0;
            if (const int rc = read_words(g, &npri, nheavy + 1, sizeof npri)) return rc;
            pr.edges = npri;
            runs.keys = sorted;
            runs.wbits = nbits;
            k_heavy_order<<<grid_for(nh, 256), 256, 0, s>>>(sorted, nh, heavy_list);
            g->launches += 2 + take_primitive_launches();
        }
    }
    // Hit masks of the heavy edges (rows layout possible): the list fill then reads the masks
    // instead of repeating the lookups.  A graph-owned buffer (reused by later counts);
    // skipped when it would take more than a third of the free memory.
    std::unique_ptr<Scratch> msc;
    int64_t* moff = nullptr;
    uint32_t* masks = nullptr;
    longlong2* pieces = nullptr;
    int64_t np[2] = {0, 0};  // pieces of the priority rows' runs, of the others
    if (rs.tab) {
        if (nh > 0) {
            msc.reset(new Scratch(g));
            int64_t* wcount = (int64_t*)msc->get(sizeof(int64_t) * (nh + 1));
            moff = (int64_t*)msc->get(sizeof(int64_t) * (nh + 1));
            int64_t* wtmp = (int64_t*)msc->get(sizeof(int64_t) * scan_temp_elems(nh + 1));
            if (!wcount || !moff || !wtmp) {
                set_error("device allocation failed (hit masks)");
                return RTR_ERR_CUDA;
            }
            k_mask_words<<<grid_for(nh + 1, 256), 256, 0, s>>>(g->offsets, g->esrc, g->nbors, g->fwd, heavy_list,
                                                                nh, rs, wcount);
            RTR_TRY(exclusive_scan_i64(wcount, moff, nh + 1, nullptr, wtmp, s));
            int64_t words = 0;
            if (const int rc = read_words(g, &words, moff + nh, sizeof(int64_t))) return rc;
            if (runs.keys && n <= (1ll << kMaxBits) && nh >= kBitsEdges) {
                const int rc = cut_runs(g, *msc, rs, nh, moff, &runs, &pieces, np);
                if (rc) return rc;
            }
            const int64_t bytes = (int64_t)sizeof(uint32_t) * (words + 1);
            if (g->rows_masks_cap >= bytes)
                masks = (uint32_t*)g->rows_masks;
            else if (bytes < (int64_t)((device_avail_bytes(g) + g->rows_masks_cap) / 3))
                masks = (uint32_t*)grow_owned(g, &g->rows_masks, &g->rows_masks_cap, bytes);
            if (masks) {
                RTR_CUDA_TRY(cudaMemsetAsync(masks, 0, (size_t)bytes, s));
            } else {
                moff = nullptr;
            }
            g->launches += 1 + take_primitive_launches();
        }
    }
    ktime_begin(g, KT_EDGE_HEAVY);
    uint16_t* parts = nullptr;
    if (nparts > 0) {
        parts = (uint16_t*)sc.get(sizeof(uint16_t) * 32 * (size_t)nparts);
        if (!parts) cudaGetLastError();  // no room: the fill intersects twice
    }
    const HeavyArgs ha{g->offsets, g->nbors, g->esrc, g->deg, g->fwd, g->partner, heavy_list, g->tune_gallop, rs, g->sup,
                       cnt, cgt, heavy_pe ? g->pe : nullptr, g->ctr, moff, masks, parts, parts ? nparts : 0};
    if (pr.count > 0 && pr.edges > 0) {
        if (const int rc = launch_bits(g, ha, runs, pieces, np[0], hq + 2)) return rc;
        k_edge_count_heavy<<<gc, kHeavyEdgeBlock, 0, s>>>(ha, runs, 0, pr.edges, nheavy, hq);
        g->launches += 1;
        const int rc = fold_priority_rows(g, sc, rs, &pr, cgt, heavy_list, moff, masks);
        if (rc) return rc;
    }
    if (const int rc = launch_bits(g, ha, runs, pieces + np[0], np[1], hq + 3)) return rc;
    k_edge_count_heavy<<<gc, kHeavyEdgeBlock, 0, s>>>(ha, runs, pr.count > 0 ? pr.edges : 0, -1, nheavy, hq + 1);
    ktime_end(g, KT_EDGE_HEAVY);
    if (rs.tab) light(nullptr);
    ktime_end(g, KT_EDGE_FOLD);
    RTR_TRY(exclusive_scan_i64(cnt, g->tl_off, m2 + 1, (int64_t*)(g->ctr + 4), tmp, s));
    g->launches += 2 + take_primitive_launches();
    RTR_CUDA_TRY(cudaGetLastError());
    unsigned long long words[2] = {0, 0};  // list entries, heavy edges (low half)
    if (const int rc = read_words(g, words, g->ctr + 4, sizeof words)) return rc;
    const int64_t tl_len = (int64_t)words[0];
    const bool heavy = (unsigned)words[1] != 0;
    bool keep_lists = g->count_mode != 2;
    if (g->count_mode == 0 && (tl_len > g->tl_len || !g->tl)) {
        // keep the lists only when they fit beside what the clean will need (records, stacks);
        // a large graph first has the pool return its cached blocks
        // free memory counts the pool's cached blocks (an earlier graph's freed buffers, which a
        // later allocation reuses) and this graph's own rows-layout buffers
        const double use = (double)sizeof(TriEntry) * (double)(tl_len + 1) + 64.0 * (double)(m + 1);
        const double own = (double)(g->rows_masks_cap + g->rows_lists_cap + g->rows_ahead_cap);
        const double margin = (double)(1ll << 30);
        // small lists may come from the pool's cached blocks alone: the device is not asked for its
        // free memory, which takes 64 us, as long as the rest of a small graph's count
        keep_lists = (use <= kListsSmall && use <= (double)pool_cached_bytes(g)) ||
                     use + margin <= (double)device_avail_bytes(g) + own;
    }
    if (keep_lists) {
        if (pr.folding) {  // the lists are kept after all: they fold every vertex
            RTR_CUDA_TRY(cudaStreamSynchronize(g->side));
            pr.folding = false;
        }
        // the rows layout's buffers are not needed with lists
        msc.reset();
        moff = nullptr;
        masks = nullptr;
        release_owned(g, &g->rows_masks, &g->rows_masks_cap);
        release_owned(g, &g->rows_lists, &g->rows_lists_cap);
        release_owned(g, &g->rows_ahead, &g->rows_ahead_cap);
        if (tl_len > g->tl_len || !g->tl) {
            // grow-only buffer owned by the graph
            TriEntry* tl = (TriEntry*)dev_alloc(g, sizeof(TriEntry) * (size_t)(tl_len + 1));
            if (tl) {
                g->tl = tl;
            } else if (g->count_mode == 0) {
                cudaGetLastError();  // less room than it looked: cached blocks in pieces, or taken by others
                keep_lists = false;
            } else {
                set_error("device allocation failed for %lld triangle-list entries", (long long)tl_len);
                return RTR_ERR_CUDA;
            }
        }
    }
    if (!keep_lists) {
        // rows layout: perVertex and heavy-edge perEdge straight from the CSR rows
        g->lists = false;
        g->tl_len = 0;
        if (!heavy_pe) {  // fold the heavy edges' perEdge now (the counts are recomputed, unchanged)
            unsigned long long* junk = (unsigned long long*)sc.get(sizeof(unsigned long long) * 2);
            if (!junk) {
                set_error("device allocation failed (count scratch)");
                return RTR_ERR_CUDA;
            }
            HeavyArgs again = ha;
            again.cgt = nullptr;
            again.pe = g->pe;
            again.total = junk;
            again.moff = nullptr;
            again.masks = nullptr;
            again.nparts = 0;
            k_edge_count_heavy<<<gc, kHeavyEdgeBlock, 0, s>>>(again, HeavyRuns{nullptr, 0, n, nullptr, nullptr}, 0, -1, nheavy,
                                                              hq + 4);
            g->launches += 1;
        }
        // cnt (scanned into tl_off above) is free: it takes the lists' offsets
        const int rc = count_rows(g, sc, rs, pr, cgt, cnt, heavy_list, nheavy, moff, masks);
        if (rc) return rc;
        RTR_CUDA_TRY(cudaGetLastError());
        cudaEventRecord(e1, s);
        RTR_CUDA_TRY(cudaEventSynchronize(e1));
        cudaEventElapsedTime(&g->ms_count, e0, e1);
        ktime_read(g, KT_EDGE_FOLD);
        ktime_read(g, KT_EDGE_LIGHT);
        ktime_read(g, KT_EDGE_HEAVY);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        g->stage = 2;
        return RTR_OK;
    }
    g->tl_len = tl_len;
    g->lists = true;
    double* terms = nullptr;
    if (kSlotsPerTerm * tl_len >= m2 && tl_len > 0) {
        terms = (double*)sc.get(sizeof(double) * (size_t)tl_len);
        if (!terms) cudaGetLastError();  // no room: the folds read the lists
    }
    const bool ahead = terms && (unsigned)words[1] >= kAheadEdges;
    cudaStream_t hs = s;  // the heavy lists'
    ktime_begin(g, KT_TRI_FILL);
    // cnt (scanned into tl_off above) is free: it takes the terms' offsets
    if (terms) RTR_TRY(exclusive_scan_i64(cgt, cnt, m2 + 1, nullptr, tmp, s));
    auto gather = [&](int lo, int hi, cudaStream_t st) {
        k_fold_gather<<<grid_for(8 * m2, kBlock), kBlock, 0, st>>>(g->esrc, g->nbors, g->partner, g->deg, lo, hi, m2,
                                                                   cgt, cnt, g->tl_off, g->tl, terms);
    };
    auto fold = [&](int lo, int hi, cudaStream_t st) {
        k_fold_terms_heavy<<<grid_for(1ll << 40, kHeavyBlock, 16), kHeavyBlock, 0, st>>>(g->offsets, cnt, n, lo, hi,
                                                                                         terms, g->pv);
    };
    const int top = INT32_MAX, cut = ahead ? g->tune_edge : top;
    cudaEvent_t filled = nullptr;
    if (ahead) {
        if (!g->side) RTR_CUDA_TRY(cudaStreamCreateWithFlags(&g->side, cudaStreamNonBlocking));
        hs = g->side;
        RTR_CUDA_TRY(cudaEventCreateWithFlags(&filled, cudaEventDisableTiming));
        side_guard.lists = filled;
        RTR_CUDA_TRY(cudaEventRecord(filled, s));
        RTR_CUDA_TRY(cudaStreamWaitEvent(hs, filled, 0));
    }
    if (heavy)
        k_tri_fill_heavy<<<gh, kHeavyEdgeBlock, 0, hs>>>(g->offsets, g->nbors, g->esrc, g->deg, g->partner, g->fwd,
                                                         g->frank, heavy_list, nheavy, g->tune_gallop, parts,
                                                         ha.nparts, g->tl_off, g->tl, hq + 5);
    if (ahead) {
        RTR_CUDA_TRY(cudaEventRecord(filled, hs));
        gather(cut, top, hs);
        fold(cut, top, hs);
        g->launches += 2;
    }
    k_tri_fill<<<ge, kBlock, 0, s>>>(g->offsets, g->nbors, g->esrc, g->deg, g->partner, g->fwd, g->frank, m,
                                     g->tl_off, g->tl, g->tune_gallop, g->tune_edge);
    if (ahead) RTR_CUDA_TRY(cudaStreamWaitEvent(s, filled, 0));
    if (heavy) k_pe_fold_heavy<<<gh, kHeavyEdgeBlock, 0, s>>>(g->fwd, heavy_list, nheavy, g->tl_off, g->tl, g->pe);
    ktime_end(g, KT_TRI_FILL);
    ktime_begin(g, KT_VERTEX_FOLD);
    if (terms) {
        gather(0, cut, s);
        k_fold_terms_light<<<grid_for(n, kBlock), kBlock, 0, s>>>(g->offsets, cnt, n, cut, terms, g->pv);
        fold(0, cut, s);
        if (ahead) {
            RTR_CUDA_TRY(cudaEventRecord(filled, hs));
            RTR_CUDA_TRY(cudaStreamWaitEvent(s, filled, 0));
        }
        g->launches += 3 + take_primitive_launches();
    } else {
        k_vertex_fold_light<<<grid_for(n, kBlock), kBlock, 0, s>>>(g->offsets, g->nbors, g->deg, g->partner, n, cgt,
                                                                    g->tl_off, g->tl, g->pv, g->tune_heavy);
        k_vertex_fold_heavy<<<grid_for(1ll << 40, kHeavyBlock, 16), kHeavyBlock, 0, s>>>(
            g->offsets, g->nbors, g->deg, g->partner, n, cgt, g->tl_off, g->tl, g->pv, g->tune_heavy);
        g->launches += 2;
    }
    ktime_end(g, KT_VERTEX_FOLD);
    g->launches += heavy ? 3 : 1;
    RTR_CUDA_TRY(cudaGetLastError());
    cudaEventRecord(e1, s);
    RTR_CUDA_TRY(cudaEventSynchronize(e1));
    cudaEventElapsedTime(&g->ms_count, e0, e1);
    ktime_read(g, KT_EDGE_FOLD);
    ktime_read(g, KT_EDGE_LIGHT);
    ktime_read(g, KT_EDGE_HEAVY);
    ktime_read(g, KT_TRI_FILL);
    ktime_read(g, KT_VERTEX_FOLD);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    g->stage = 2;
    return RTR_OK;
}

}  // namespace rtr
