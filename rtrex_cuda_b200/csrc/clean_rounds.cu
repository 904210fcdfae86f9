// Window replay of a large clean unit, order-faithful to initialClean +
// deleteAndClean (RTRex_Sequential/Escape/Decomposition.h:302-460, :147-283).
//
// The reference pops one edge at a time from a LIFO stack; a pop reads and
// writes only the records of its own edge and of the other two edges of each
// of its live triangles ("cells"), and the perVertex weights of the
// triangles' vertices -- which no pop ever reads.  As long as no pop pushes,
// the order of the next pops is known: the stack from its top, then the seeds.
// One thread block replays one unit in rounds, each over the window of the
// next items in that order (at most W items whose triangle lists fit the
// block's threads, one list entry per thread):
//
//  1. an entry's triangle is live for its item unless one of the other two
//     edges is already deleted or is itself an earlier item of the window;
//  2. every live triangle subtracts its weight from its two other edges.  A
//     direct-mapped table in shared memory (per slot: a mask of the items that
//     use it, and per item which thread's triangle and which of its edges)
//     shows each thread the earlier items that subtract from its edges; it
//     applies those in item order, then its own, and checks the threshold, as
//     the reference does;
//  3. the first item after which some edge falls below its threshold (the
//     first item that pushes) ends the window: it and the items before it are
//     committed -- their values are those of the sequential replay -- and the
//     later items' subtractions are dropped;
//  4. the committed items leave the stack and the pusher's pushes go on top,
//     in the reference's push order (triangle order, (lower,w) before
//     (higher,w)).
//
// Where nearly every pop pushes, a window commits one or two items and costs as
// much as a full one.  Units of few seeds for their edges, whose pops are mostly
// pushed ones, therefore take a form (kOne) that watches the pops a round commits
// and, while they are few, lets the first warp pop items one by one.
//
// So the committed pops come in exactly the reference's order.  Each is logged
// with its number of live triangles, and a byte per list entry says which of
// them the pop removed.  After the replay the popped edges' own perEdge and the
// perVertex subtractions are folded from that log: k_log_keys numbers the
// removed triangles in pop order and writes their (vertex, number) keys, a
// stable radix sort groups them by vertex, k_log_gather / k_fold_long_runs
// subtract each vertex's weights in that order.
//
// What bounds it: a round is one dependent chain (window, entries, records,
// table, fold, commit; 4 barriers) of ~4,000 cycles, of which the memory is a
// fifth and the rest instruction latency, and every item that pushes ends a
// round.  On the 926,000-edge co-purchase graph (B200, eps 0.3) the giant
// unit's 41,800 pops take 7,340 rounds (5,440 ended by a push), 14.4 ms; reserving
// cells and letting only conflict-free items commit (with the sequence as a linked
// list, ranked afterwards) took 25.0 ms, one warp per unit 38.5 ms.  On the
// 203,311-edge R-MAT graph (mean list 31) 162,000 pops take 40,700 rounds (25,700
// ended by a push), 111 ms against 235 ms one warp per unit.  Measured and slower:
// a warp replaying single items from lists brought into L1 by helper warps (19.7 /
// 203 ms), one thread per edge folding all items' subtractions (18.9 / 148 ms), one
// warp walking the window's items in shared memory after a parallel load (27.5 /
// 139 ms).
//
// An item whose list does not fit is popped alone, its entries taken one block
// width at a time.
#include "clean_units.cuh"
#include "fold_run.cuh"
#include "primitives.cuh"
#include "rtr_graph.cuh"

#include <algorithm>

namespace rtr {

namespace {

constexpr int kBlock = 256;
constexpr unsigned kFull = 0xffffffffu;
constexpr int kLow = 64;  // stack entries below which the ring is refilled (more than a window)
constexpr int kOwnBits = 10;
constexpr int kOwnSlots = 1 << kOwnBits;

// NW warps, one list entry per thread.  G > 0: G threads for each item (a longer
// list is popped alone); G == 0: the items' lists packed back to back.
template <int NW, int G, int W>
struct Cfg {
    static constexpr int kThreads = 32 * NW;
    static constexpr int kSlots = NW <= 8 ? 1024 : 2048;
    static constexpr int kRing = NW <= 8 ? 1024 : 2048;
    static constexpr int kSpare = 1 << 7;  // slots for an item's second edge in one slot
    static constexpr int kAll = kSlots + W + kSpare;
    static_assert(G == 0 || kThreads == G * W, "G threads per window item");
    static_assert(kLow + 3 * kThreads <= kRing, "a refill and a window's pushes fit the ring");
};

// A live triangle's subtraction from one of its two other edges.
struct alignas(16) Sub {
    double w;
    unsigned cell;  // the edge
    int next;       // the next window item that subtracts from it (W: none; item | 32: that item pops it)
};

template <int NW, int G, int W>
struct WinSmem {
    using C = Cfg<NW, G, W>;
    StackEntry ring[C::kRing];                  // the newest stack entries, circular
    Sub sub[2 * C::kThreads + 1];               // the two subtractions of each thread's live triangle (last: none)
    uint16_t hid[C::kAll * W];               // which one is in a slot, per item (valid under hmask)
    unsigned hmask[C::kAll];                    // window items in a slot ([kSlots, kSlots + W): their own edges)
    unsigned twice;                             // items with an edge in a spare slot
    unsigned own[kOwnSlots];                    // the window's own edges: tag | item + 1
    int wpush[NW];
    int wlive[NW];
    int cut[2];                                 // where the window ends, by round parity (see below)
    int npush;
    int2 single;                                // where a run of single pops left the stack's top, and its pops
};

struct RoundArgs {
    const TriEntry* tl;
    EdgeRec* rec;
    double inv_n;
    const StackEntry* seeds;
    const UnitDesc* units;
    const uint64_t* order;  // the launch's units
    StackEntry* stacks;
    PopLog* plog;    // pops of each unit from its stack_base
    uint8_t* live8;  // per list entry: its triangle was removed by the pop of its list's edge
    unsigned* err;
    unsigned long long* total;
    unsigned long long* diag;
};

// An edge's weight, list length and support word (the first half of its record) in one store.
__device__ __forceinline__ void store_state(EdgeRec* p, const EdgeRec& r)
{
    *reinterpret_cast<int4*>(p) = *reinterpret_cast<const int4*>(&r);
}

__device__ __forceinline__ void load_state(const EdgeRec* p, EdgeRec& r)
{
    *reinterpret_cast<int4*>(&r) = *reinterpret_cast<const int4*>(p);
}

// A cut value: the window ends with item `last`, which pushes (2 * last) or
// after which the later items may not be taken (2 * last + 1).
__device__ __forceinline__ int cut_after(int last) { return 2 * (last > 0 ? last : 0) + 1; }

// Pops one by one (kOne): after kTries rounds that committed fewer than kWorth pops
// each on average (a round takes ~4,000 cycles, a warp's pop ~2,000), the first
// warp takes the next kSingleFirst pops, twice as many each time the windows are
// found wanting again, kSingleMost at most.  Rounds that a list of more than
// kSingleList entries ends or fills say nothing: such an item is the block's.
// Windows alone / with single pops / one warp per unit, ms: triangular lattice
// (186,501 edges, 996 seeds) 216 / 121 / 142, Delaunay mesh (149,970) 138 / 91 / 102,
// points in the plane of mean degree 20 (98,385, eps 0.5) 66 / 46 / 64, in space of
// 25 (112,529, eps 0.3) 71 / 50 / 61; where windows do well it costs 2 to 3%.
constexpr int kTries = 16;
constexpr int kWorth = 2;
constexpr int kSingleFirst = 64, kSingleMost = 4096;
constexpr int kSingleList = 64;

// The first 16 entries of a list that a later round reads: into L1 as soon as an
// edge is seen to fall (its push is likely the next round's first item), into L2
// when a seed enters the ring.  Co-purchase graph 15.6 -> 14.8 with the first, 14.4
// ms with both; R-MAT 203,311 edges 117.3 -> 112.5 -> 111.5, 40,000 20.3 -> 19.5 -> 19.5.
// (Whole lists by bulk prefetch at the push: 112 and 15.2 ms, but 21.0 for 40,000
// edges -- issuing one costs the round 200 cycles.  In k_clean_units, where one warp
// issues everything, the same prefetches cost 3 to 11%.)
constexpr int kTouch = 4;  // lines of 4 entries

__device__ __forceinline__ void touch_list(const TriEntry* p, int32_t cnt)
{
#pragma unroll
    for (int k = 0; k < kTouch; ++k)
        if (4 * k < cnt) asm volatile("prefetch.global.L1 [%0];" ::"l"(p + 4 * k));
}

__device__ __forceinline__ void ask_list(const TriEntry* p, int32_t cnt)
{
#pragma unroll
    for (int k = 0; k < kTouch; ++k)
        if (4 * k < cnt) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + 4 * k));
}

constexpr int kSpareBits = 7;
__device__ __forceinline__ int spare_hash(unsigned cell) { return (int)((cell * 2654435761u) >> (32 - kSpareBits)); }

// An edge's weight after the subtractions of the items in `lower` (ascending);
// counts them and names the last one.  `twice`: items with an edge in a spare slot.
template <int NW, int G, int W>
__device__ __forceinline__ double fold_lower(const WinSmem<NW, G, W>& S, int slot, unsigned lower, unsigned twice,
                                             unsigned cell, double x, uint32_t& n, int& prev)
{
    if (lower & twice) {
        for (unsigned l = lower; l; l &= l - 1) {
            const int q = __ffs(l) - 1;
            int id = S.hid[slot * W + q];
            if (S.sub[id].cell != cell && ((twice >> q) & 1u)) {
                const int z = Cfg<NW, G, W>::kSlots + W + spare_hash(cell);
                if ((S.hmask[z] >> q) & 1u) id = S.hid[z * W + q];
            }
            if (S.sub[id].cell == cell) {
                x -= S.sub[id].w;
                ++n;
                prev = id;
            }
        }
        return x;
    }
    const uint4* row = reinterpret_cast<const uint4*>(&S.hid[slot * W]);
#pragma unroll
    for (int b = 0; b < W; b += 8) {
        if (((lower >> b) & 255u) == 0) continue;
        const uint4 v = row[b / 8];
        const unsigned r[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
            // four items' subtractions loaded together
            if (((lower >> (b + h)) & 15u) == 0) continue;
            int id[4];
            Sub u[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                id[k] = (int)((r[(h + k) >> 1] >> (16 * (k & 1))) & 0xffffu);
                u[k] = S.sub[(lower >> (b + h + k)) & 1u ? id[k] : 2 * Cfg<NW, G, W>::kThreads];
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const bool hit = u[k].cell == cell;
                x = hit ? x - u[k].w : x;
                n += hit ? 1u : 0u;
                prev = hit ? id[k] : prev;
            }
        }
    }
    return x;
}

struct SinglePops {
    int top, done;
    unsigned long long removed;
};

// The first warp's pops, at most n, from the ring positions [bot, top).  Out of
// line: the rounds' own code then stays as it is without it.
template <int R>
__device__ __noinline__ SinglePops pop_singles(const TriEntry* tl, EdgeRec* rec, PopLog* plog, uint8_t* live8,
                                               StackEntry* ring, int top, int bot, int n)
{
    constexpr int M = R - 1;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    int done = 0;
    unsigned long long removed = 0;
    while (done < n && top > bot) {
        const StackEntry c = ring[(top - 1) & M];
        if (c.cnt > kSingleList || top - 1 - bot + 2 * c.cnt > R) break;
        __syncwarp();  // c is read before a push takes its place
        const PairSide ps = pair_side(c);
        TriEntry t{};
        if (lane < c.cnt) t = ld_entry(tl + c.t0 + lane);
        const uint32_t s_e = rec[c.e].ss & SS_SUP;
        top -= 1;
        for (int base = 0; base < c.cnt && s_e > 0; base += 32) {
            const bool valid = base + lane < c.cnt;
            if (base > 0 && valid) t = ld_entry(tl + c.t0 + base + lane);
            EdgeRec r1{}, r2{};
            r1.ss = r2.ss = SS_N;
            const int32_t rlw = ps.lower_is_a ? t.raz : t.rbz;
            const int32_t rhw = ps.lower_is_a ? t.rbz : t.raz;
            if (valid) {
                r1 = rec[rlw];
                r2 = rec[rhw];
            }
            const uint32_t c1 = r1.ss & SS_CODE, c2 = r2.ss & SS_CODE;
            bool f1 = false, f2 = false;
            if (valid && c1 != SS_N && c2 != SS_N) {
                r1.pe -= t.wgt;
                r2.pe -= t.wgt;
                f1 = c1 != SS_S && r1.pe < r1.thr;
                f2 = c2 != SS_S && r2.pe < r2.thr;
                r1.ss = ((r1.ss & SS_SUP) - 1u) | (f1 ? SS_S : c1);
                r2.ss = ((r2.ss & SS_SUP) - 1u) | (f2 ? SS_S : c2);
                store_state(rec + rlw, r1);
                store_state(rec + rhw, r2);
                live8[c.t0 + base + lane] = 1;
                if (f1) touch_list(tl + r1.t0, (int32_t)r1.cnt);
                if (f2) touch_list(tl + r2.t0, (int32_t)r2.cnt);
            }
            const unsigned b1 = __ballot_sync(kFull, f1), b2 = __ballot_sync(kFull, f2);
            const int q = top + __popc(b1 & lt) + __popc(b2 & lt);
            if (f1) ring[q & M] = StackEntry{rlw, ps.lower, t.z, ps.dlow, t.dz, (int32_t)r1.cnt, r1.t0};
            if (f2)
                ring[(q + (f1 ? 1 : 0)) & M] = StackEntry{rhw, ps.higher, t.z, ps.dhigh, t.dz, (int32_t)r2.cnt, r2.t0};
            top += __popc(b1) + __popc(b2);
        }
        if (lane == 0) {
            rec[c.e].ss = SS_N;  // every live triangle of it is gone
            plog[done] = PopLog{c.e, (int32_t)s_e, c.t0};
        }
        removed += s_e;
        __syncwarp();
        ++done;
    }
    return SinglePops{top, done, removed};
}

template <int NW, int G, int W, bool kOne>
__global__ void __launch_bounds__(32 * NW) k_clean_rounds(RoundArgs a)
{
    using C = Cfg<NW, G, W>;
    constexpr int T = C::kThreads;
    constexpr int M = C::kRing - 1;
    constexpr int H = C::kSlots;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    WinSmem<NW, G, W>& S = *reinterpret_cast<WinSmem<NW, G, W>*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const UnitDesc ud = a.units[(uint32_t)a.order[blockIdx.x]];
    StackEntry* gm = a.stacks + ud.stack_base;
    PopLog* plog = a.plog + ud.stack_base;
    for (int i = tid; i < C::kAll; i += T) S.hmask[i] = 0;
    for (int i = tid; i < kOwnSlots; i += T) S.own[i] = 0;
    if (tid < 2) S.cut[tid] = cut_after(W);
    if (tid == 0) {
        S.twice = 0;
        S.sub[2 * T].cell = ~0u;
    }
    // The stack, identical in every thread: ring positions [bot, top) (top - 1 =
    // next), below them the unit's global region gm[0, gtop), below it the
    // seeds [seed_begin, sp).
    int top = 1 << 28, bot = 1 << 28;
    int64_t gtop = 0, sp = ud.seed_end;
    int64_t npop = 0;
    unsigned long long removed = 0;  // of this thread's items
    int par = 0;
    bool fail = false;
    int single = 0, hold = kSingleFirst;  // pops to take one by one; how many the next time
    int tried = 0, taken = 0;             // window rounds since the last decision, and their pops
    __syncthreads();
    // the oldest `s` ring entries to the global region
    auto spill = [&](int s) {
        if (gtop + s > ud.stack_cap) {
            if (tid == 0) atomicOr(a.err, (unsigned)DEV_ERR_STACK_OVERFLOW);
            fail = true;
            return;
        }
        for (int j = tid; j < s; j += T) gm[gtop + j] = S.ring[(bot + j) & M];
        gtop += s;
        bot += s;
        __syncthreads();
    };
    while (true) {
        while (top - bot < kLow && (gtop > 0 || sp > ud.seed_begin)) {
            if (gtop > 0) {
                const int k = (int)(gtop < T ? gtop : T);
                if (tid < k) S.ring[(bot - 1 - tid) & M] = gm[gtop - 1 - tid];
                gtop -= k;
                bot -= k;
            } else {
                // Seeds whose support is already 0 are retired here without a
                // pop: support only decreases, and such a pop touches no cell
                // but its own and pushes nothing.
                const int k = (int)(sp - ud.seed_begin < T ? sp - ud.seed_begin : T);
                StackEntry se{};
                bool kept = tid < k;
                if (kept) {
                    se = a.seeds[sp - 1 - tid];
                    const EdgeRec* x = a.rec + se.e;
                    const double pe = x->pe;
                    kept = (x->ss & SS_SUP) > 0;
                    if (!kept) {
                        if (fabs(pe) > a.inv_n) atomicAdd(a.diag, 1ull);
                        a.rec[se.e].ss = SS_N;
                    }
                }
                const unsigned bal = __ballot_sync(kFull, kept);
                if (lane == 0) S.wlive[wid] = __popc(bal);
                __syncthreads();
                const int x = lane < NW ? S.wlive[lane] : 0;
                const int below = __reduce_add_sync(kFull, lane < wid ? x : 0);
                if (kept) {
                    ask_list(a.tl + se.t0, se.cnt);
                    S.ring[(bot - 1 - below - __popc(bal & lt)) & M] = se;
                }
                sp -= k;
                bot -= __reduce_add_sync(kFull, x);
            }
            __syncthreads();
        }
        const int avail = top - bot;
        if (avail <= 0) break;
        if (npop >= ud.edges) {  // every edge of the unit has been popped: the stack must be empty
            if (tid == 0) atomicOr(a.err, (unsigned)DEV_ERR_BAD_STATUS);
            break;
        }
        if (avail > C::kRing - 2 * T) {  // room for a round's pushes
            spill(avail - (C::kRing - 2 * T) + C::kRing / 4);
            if (fail) break;
        }
        // ---- one by one, by the first warp
        if (kOne && single > 0) {
            if (wid == 0) {
                const int64_t left = ud.edges - npop;
                const SinglePops p = pop_singles<C::kRing>(a.tl, a.rec, plog + npop, a.live8, S.ring, top, bot,
                                                           left < single ? (int)left : single);
                if (lane == 0) {
                    S.single = make_int2(p.top, p.done);
                    removed += p.removed;
                }
            }
            __syncthreads();
            const int2 s = S.single;
            __syncthreads();  // read before the first warp writes it again
            top = s.x;
            npop += s.y;
            single -= s.y;
            if (s.y > 0) continue;  // else the next item's list is the block's
        }
        // ---- the window: this thread's item and list entry
        int ni = avail < W ? avail : W;
        int item, j;
        bool alone;
        int i0 = 0, i1 = 0;  // G == 0: lane k holds the first and one-past-last entry of item k
        if (G > 0) {
            item = tid / (G > 0 ? G : 1);
            j = tid % (G > 0 ? G : 1);
            alone = S.ring[(top - 1) & M].cnt > G;
        } else {
            const int cnt = lane < ni ? S.ring[(top - 1 - lane) & M].cnt : 0;
            i1 = cnt;
#pragma unroll
            for (int o = 1; o < W; o <<= 1) {
                const int y = __shfl_up_sync(kFull, i1, o);
                if (lane >= o) i1 += y;
            }
            i0 = i1 - cnt;
            const bool fit = cnt > 0 && i1 <= T;
            ni = __popc(__ballot_sync(kFull, fit));
            alone = ni == 0;
            const int rel = i0 - 32 * wid;
            const unsigned here = __reduce_or_sync(kFull, fit && rel >= 0 && rel < 32 ? 1u << rel : 0u);
            const int before = __popc(__ballot_sync(kFull, fit && rel < 0));
            item = before + __popc(here & (lt | (1u << lane))) - 1;
            j = tid - __shfl_sync(kFull, i0, item & 31);
        }
        if (alone) {
            // ---- a list longer than the window takes: popped alone, one block width at a
            // time (within one pop the cells of its triangles are distinct)
            const StackEntry c = S.ring[(top - 1) & M];
            const PairSide ps = pair_side(c);
            const uint32_t s_e = a.rec[c.e].ss & SS_SUP;
            top -= 1;
            __syncthreads();  // c is read before a push takes its place
            for (int base = 0; base < c.cnt && s_e > 0; base += T) {
                const bool valid = base + tid < c.cnt;
                TriEntry t{};
                EdgeRec r1{}, r2{};
                r1.ss = r2.ss = SS_N;
                if (valid) t = ld_entry(a.tl + c.t0 + base + tid);
                const int32_t rlw = ps.lower_is_a ? t.raz : t.rbz;
                const int32_t rhw = ps.lower_is_a ? t.rbz : t.raz;
                if (valid) {
                    r1 = a.rec[rlw];
                    r2 = a.rec[rhw];
                }
                const uint32_t c1 = r1.ss & SS_CODE, c2 = r2.ss & SS_CODE;
                const bool live = valid && c1 != SS_N && c2 != SS_N;
                bool f1 = false, f2 = false;
                if (live) {
                    const double x1 = r1.pe - t.wgt, x2 = r2.pe - t.wgt;
                    f1 = c1 != SS_S && x1 < r1.thr;
                    f2 = c2 != SS_S && x2 < r2.thr;
                    a.rec[rlw].pe = x1;
                    a.rec[rhw].pe = x2;
                    a.rec[rlw].ss = ((r1.ss & SS_SUP) - 1u) | (f1 ? SS_S : c1);
                    a.rec[rhw].ss = ((r2.ss & SS_SUP) - 1u) | (f2 ? SS_S : c2);
                    a.live8[c.t0 + base + tid] = 1;
                }
                const unsigned b1 = __ballot_sync(kFull, f1), b2 = __ballot_sync(kFull, f2);
                if (lane == 0) S.wpush[wid] = __popc(b1) + __popc(b2);
                __syncthreads();
                const int x = lane < NW ? S.wpush[lane] : 0;
                const int ppre = __reduce_add_sync(kFull, lane < wid ? x : 0);
                const int pall = __reduce_add_sync(kFull, x);
                if (top - bot + pall > C::kRing) {
                    spill(top - bot + pall - C::kRing + C::kRing / 4);
                    if (fail) break;
                }
                const int p = top + ppre + __popc(b1 & lt) + __popc(b2 & lt);
                if (f1) S.ring[p & M] = StackEntry{rlw, ps.lower, t.z, ps.dlow, t.dz, (int32_t)r1.cnt, r1.t0};
                if (f2)
                    S.ring[(p + (f1 ? 1 : 0)) & M] =
                        StackEntry{rhw, ps.higher, t.z, ps.dhigh, t.dz, (int32_t)r2.cnt, r2.t0};
                top += pall;
                __syncthreads();
            }
            if (fail) break;
            if (tid == 0) {
                a.rec[c.e].ss = SS_N;  // every live triangle of it is gone
                plog[npop] = PopLog{c.e, (int32_t)s_e, c.t0};
                removed += s_e;
            }
            npop += 1;
            __syncthreads();
            continue;
        }
        // ---- the item, its entry, the two other records of the entry's triangle
        StackEntry c{};
        bool valid = item < ni;
        if (valid) c = S.ring[(top - 1 - item) & M];
        int cut = cut_after(W);  // this thread's bound on the window's end
        if (G > 0 && valid && c.cnt > G) cut = cut_after(item - 1);
        valid = valid && j < c.cnt && (G == 0 || c.cnt <= G);
        const bool owner = valid && j == 0;
        const unsigned own_tag = (((unsigned)c.e >> kOwnBits) << 5) | (unsigned)(item + 1);
        TriEntry t{};
        EdgeRec r1{}, r2{};  // the first halves; thr and t0 are read only where they are needed
        r1.ss = r2.ss = SS_N;
        uint32_t oss = 0;
        const PairSide ps = pair_side(c);
        int32_t rlw = 0, rhw = 0;
        if (valid) {
            t = ld_entry(a.tl + c.t0 + j);
            if (owner) {
                S.own[(unsigned)c.e & (kOwnSlots - 1)] = own_tag;
                oss = a.rec[c.e].ss;
            }
            rlw = ps.lower_is_a ? t.raz : t.rbz;
            rhw = ps.lower_is_a ? t.rbz : t.raz;
            load_state(a.rec + rlw, r1);
            load_state(a.rec + rhw, r2);
        }
        __syncthreads();  // A: the window's own edges are in S.own
        if (tid == 0) S.cut[par ^ 1] = cut_after(W);
        const uint32_t c1 = r1.ss & SS_CODE, c2 = r2.ss & SS_CODE;
        const unsigned bit = 1u << item;
        // an own edge displaced from S.own by another item's: the window ends before it
        if (owner && S.own[(unsigned)c.e & (kOwnSlots - 1)] != own_tag) cut = cut_after(item - 1);
        int s1 = 0, s2 = 0;
        bool live = valid && c1 != SS_N && c2 != SS_N;
        if (live) {
            const unsigned o1 = S.own[(unsigned)rlw & (kOwnSlots - 1)], o2 = S.own[(unsigned)rhw & (kOwnSlots - 1)];
            const int q1 = o1 != 0 && (o1 >> 5) == (unsigned)rlw >> kOwnBits ? (int)(o1 & 31u) - 1 : W;
            const int q2 = o2 != 0 && (o2 >> 5) == (unsigned)rhw >> kOwnBits ? (int)(o2 & 31u) - 1 : W;
            s1 = q1 < W ? H + q1 : rlw & (H - 1);
            s2 = q2 < W ? H + q2 : rhw & (H - 1);
            live = q1 > item && q2 > item;  // else deleted by an earlier item of the window
        }
        int z1 = 0, z2 = 0;  // spare slots taken
        if (live) {
            if (c1 != SS_S) r1.thr = a.rec[rlw].thr;
            if (c2 != SS_S) r2.thr = a.rec[rhw].thr;
            S.sub[2 * tid] = Sub{t.wgt, (unsigned)rlw, W};
            S.sub[2 * tid + 1] = Sub{t.wgt, (unsigned)rhw, W};
            const unsigned b1 = atomicOr(&S.hmask[s1], bit), b2 = atomicOr(&S.hmask[s2], bit);
            // another edge of this item has the slot: a spare slot, or the window ends before the item
            if (b1 & bit) {
                z1 = H + W + spare_hash((unsigned)rlw);
                atomicOr(&S.twice, bit);
                if (atomicOr(&S.hmask[z1], bit) & bit) cut = cut_after(item - 1);
            }
            if (b2 & bit) {
                z2 = H + W + spare_hash((unsigned)rhw);
                atomicOr(&S.twice, bit);
                if (atomicOr(&S.hmask[z2], bit) & bit) cut = cut_after(item - 1);
            }
            S.hid[(z1 ? z1 : s1) * W + item] = (uint16_t)(2 * tid);
            S.hid[(z2 ? z2 : s2) * W + item] = (uint16_t)(2 * tid + 1);
        }
        __syncthreads();  // B: every subtraction is in the table
        double x1 = 0.0, x2 = 0.0;
        uint32_t n1 = 1, n2 = 1;
        bool f1 = false, f2 = false;
        unsigned om = 0;  // earlier items that subtract from the owner's own edge
        if (owner) {
            om = S.hmask[H + item];
            if (om) S.sub[S.hid[(H + item) * W + 31 - __clz(om)]].next = item | 32;
        }
        if (live) {
            // fold this thread's two cells through its own item: the earlier items'
            // subtractions in item order, then its own
            const unsigned l1 = S.hmask[s1] & (bit - 1u), l2 = S.hmask[s2] & (bit - 1u);
            const unsigned tw = S.twice;
            x1 = r1.pe;
            x2 = r2.pe;
            int p1 = -1, p2 = -1;
            if (l1) x1 = fold_lower<NW, G, W>(S, s1, l1, tw, (unsigned)rlw, x1, n1, p1);
            if (l2) x2 = fold_lower<NW, G, W>(S, s2, l2, tw, (unsigned)rhw, x2, n2, p2);
            if (p1 >= 0) S.sub[p1].next = item;
            if (p2 >= 0) S.sub[p2].next = item;
            x1 -= t.wgt;
            x2 -= t.wgt;
            f1 = c1 != SS_S && x1 < r1.thr;
            f2 = c2 != SS_S && x2 < r2.thr;
            if ((f1 || f2) && 2 * item < cut) cut = 2 * item;
            if (f1) touch_list(a.tl + a.rec[rlw].t0, (int32_t)r1.cnt);
            if (f2) touch_list(a.tl + a.rec[rhw].t0, (int32_t)r2.cnt);
        }
        cut = __reduce_min_sync(kFull, cut);
        if (lane == 0 && cut < cut_after(W)) atomicMin(&S.cut[par], cut);
        __syncthreads();  // C: the window's end is known
        cut = S.cut[par];
        if (cut > 2 * ni - 1) cut = 2 * ni - 1;
        const int last = cut >> 1;
        const bool pushed = (cut & 1) == 0;
        if (live) {
            S.hmask[s1] = 0;
            S.hmask[s2] = 0;
            if (z1) S.hmask[z1] = 0;
            if (z2) S.hmask[z2] = 0;
            if (item <= last) {
                // the last committed item that subtracts from a cell stores it; the
                // status of an edge that is itself popped is its owner's to store
                const int y1 = S.sub[2 * tid].next, y2 = S.sub[2 * tid + 1].next;
                r1.pe = x1;
                r1.ss = (y1 & 31) > last ? ((r1.ss & SS_SUP) - n1) | (f1 ? SS_S : c1) : SS_N;
                r2.pe = x2;
                r2.ss = (y2 & 31) > last ? ((r2.ss & SS_SUP) - n2) | (f2 ? SS_S : c2) : SS_N;
                if (y1 > last) store_state(a.rec + rlw, r1);
                if (y2 > last) store_state(a.rec + rhw, r2);
                a.live8[c.t0 + j] = 1;
            }
        }
        if (tid == 0) S.twice = 0;
        if (owner) {
            // its pop leaves it without a live triangle
            S.own[(unsigned)c.e & (kOwnSlots - 1)] = 0;
            if (item <= last) {
                const uint32_t left = (oss & SS_SUP) - (uint32_t)__popc(om);
                if (!om) a.rec[c.e].ss = SS_N;
                if (npop + item < ud.edges) plog[npop + item] = PopLog{c.e, (int32_t)left, c.t0};
                removed += left;
            }
        }
        int npush = 0, last_cnt = 0;
        if (pushed) {
            // its pushes in the reference's order, from ring position top - (last + 1)
            const bool mine = live && item == last;
            const unsigned b1 = __ballot_sync(kFull, mine && f1), b2 = __ballot_sync(kFull, mine && f2);
            npush = __popc(b1) + __popc(b2);
            int base = 0, w0 = last * G >> 5, w1 = w0;
            if (G == 0) {
                const int e0 = __shfl_sync(kFull, i0, last), e1 = __shfl_sync(kFull, i1, last);
                w0 = e0 >> 5;
                w1 = (e1 - 1) >> 5;
                last_cnt = e1 - e0;
            }
            if (w0 != w1) {  // the item spans warps
                if (lane == 0) S.wpush[wid] = npush;
                __syncthreads();
                const int x = lane < NW ? S.wpush[lane] : 0;
                base = __reduce_add_sync(kFull, lane < wid ? x : 0);
                npush = __reduce_add_sync(kFull, x);
            } else if (wid == w0 && lane == 0) {
                S.npush = npush;
            }
            if (mine) {
                const int p = top - (last + 1) + base + __popc(b1 & lt) + __popc(b2 & lt);
                if (f1)
                    S.ring[p & M] =
                        StackEntry{rlw, ps.lower, t.z, ps.dlow, t.dz, (int32_t)r1.cnt, a.rec[rlw].t0};
                if (f2)
                    S.ring[(p + (f1 ? 1 : 0)) & M] =
                        StackEntry{rhw, ps.higher, t.z, ps.dhigh, t.dz, (int32_t)r2.cnt, a.rec[rhw].t0};
            }
            __syncthreads();  // D: records, ring and push count are in place
            if (w0 == w1) npush = S.npush;
        } else {
            __syncthreads();  // D
        }
        npop += last + 1;
        top += npush - (last + 1);
        par ^= 1;
        if (kOne && (pushed ? last_cnt <= kSingleList : last + 1 >= kWorth)) {
            taken += last + 1;
            ++tried;
        }
        if (kOne && tried == kTries) {
            if (taken < kWorth * kTries) {
                single = hold;
                hold = hold < kSingleMost ? 2 * hold : hold;
            } else {
                hold = kSingleFirst;
            }
            tried = taken = 0;
        }
    }
    if (removed) atomicAdd(a.total, (unsigned long long)(-(long long)removed));
}

// Live triangles of each pop.
__global__ void k_pop_counts(const PopLog* __restrict__ plog, int64_t cap, uint32_t* __restrict__ cnt)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < cap; i += (int64_t)gridDim.x * blockDim.x) {
        const PopLog p = plog[i];
        cnt[i] = p.e >= 0 ? (uint32_t)p.n : 0u;
    }
}

// Eight lanes per pop, its list entries eight at a time: the removed triangles
// are numbered in pop order and, within a pop, in triangle order; each one's
// weight goes to wlog and its three vertices' sort keys (vertex, number) to keys.
// The popped edge's own perEdge -- its record holds the value at the pop -- loses
// their weights in that order (deleteAndClean's own fold,
// Decomposition.h:152-281), followed by the reference's residual check; no pop
// reads a popped edge's perEdge (its triangles are no longer live).
__global__ void k_log_keys(EdgeRec* __restrict__ rec, const PopLog* __restrict__ plog,
                           const uint32_t* __restrict__ off, int64_t cap, const TriEntry* __restrict__ tl,
                           const uint8_t* __restrict__ live8, const int32_t* __restrict__ fwd,
                           const int32_t* __restrict__ esrc, const int32_t* __restrict__ nb, double inv_n, int lb,
                           uint64_t* __restrict__ keys, double* __restrict__ wlog, unsigned* __restrict__ err,
                           unsigned long long* __restrict__ diag)
{
    const int lane = threadIdx.x & 31, sub = lane & 7, g0 = lane & 24;
    const int64_t step = ((int64_t)gridDim.x * blockDim.x) >> 3;
    const int64_t rounds = (cap + step - 1) / step;
    int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 3;
    for (int64_t r = 0; r < rounds; ++r, i += step) {
        PopLog p{-1, 0, 0};
        if (i < cap) p = plog[i];
        const bool use = p.e >= 0;
        int cnt = 0;
        uint64_t L = 0, u = 0, v = 0;
        double x = 0.0;
        if (use) x = rec[p.e].pe;
        if (use && p.n > 0) {
            cnt = (int)rec[p.e].cnt;
            L = off[i];
            const int64_t s = fwd[p.e];
            u = (uint64_t)esrc[s] << lb;
            v = (uint64_t)nb[s] << lb;
        }
        int left = use ? p.n : 0;
        for (int b = 0; __any_sync(kFull, b < cnt); b += 8) {
            const bool live = b + sub < cnt && live8[p.at + b + sub] != 0;
            int32_t z = 0;
            double w = 0.0;
            if (live) {
                const TriEntry* t = tl + p.at + b + sub;
                z = t->z;
                w = t->wgt;
            }
            const unsigned m = (__ballot_sync(kFull, live) >> g0) & 0xffu;
            if (live) {
                const uint64_t at = L + (uint64_t)__popc(m & ((1u << sub) - 1u));
                if (left >= __popc(m)) {
                    wlog[at] = w;
                    keys[3 * at] = u | at;
                    keys[3 * at + 1] = v | at;
                    keys[3 * at + 2] = ((uint64_t)z << lb) | at;
                }
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) x -= __shfl_sync(kFull, w, g0 + k);  // a dead entry subtracts +0.0
            L += (uint64_t)__popc(m);
            left -= __popc(m);
        }
        if (use && sub == 0) {
            if (left != 0) atomicOr(err, (unsigned)DEV_ERR_BAD_STATUS);  // support and live triangles disagree
            rec[p.e].pe = x;
            if (fabs(x) > inv_n) atomicAdd(diag, 1ull);
        }
    }
}

constexpr int64_t kLongRun = 32;  // subtractions of one vertex from which a warp folds them

// The weights in sorted order, and the vertices' runs: a short one is folded
// here by the thread at its head, a long one queued for a warp.
__global__ void k_log_gather(const uint64_t* __restrict__ keys, int64_t cnt, int64_t n, int lb,
                             const double* __restrict__ wlog, double* __restrict__ ws, double* __restrict__ pv,
                             longlong2* __restrict__ runs, unsigned* __restrict__ nruns)
{
    const uint64_t lmask = (1ull << lb) - 1;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t key = keys[i];
        const int64_t v = (int64_t)(key >> lb);
        if (v >= n || key == ~0ull) continue;
        ws[i] = wlog[key & lmask];
        if (i > 0 && (int64_t)(keys[i - 1] >> lb) == v) continue;
        int64_t lo = i + 1, hi = cnt;  // the run's end
        if (i + kLongRun < cnt && (int64_t)(keys[i + kLongRun] >> lb) == v) lo = i + kLongRun + 1;
        else if (hi > i + kLongRun) hi = i + kLongRun;
        while (lo < hi) {
            const int64_t mid = (lo + hi) >> 1;
            if ((int64_t)(keys[mid] >> lb) == v) lo = mid + 1;
            else hi = mid;
        }
        if (lo - i > kLongRun) {
            runs[atomicAdd(nruns, 1u)] = make_longlong2(i, lo);
            continue;
        }
        double x = pv[v];
        for (int64_t k = i; k < lo; ++k) x -= wlog[keys[k] & lmask];
        pv[v] = x;
    }
}

// A warp per long run.
__global__ void __launch_bounds__(128) k_fold_long_runs(const longlong2* __restrict__ runs,
                                                        const unsigned* __restrict__ nruns,
                                                        const uint64_t* __restrict__ keys, int lb,
                                                        const double* __restrict__ ws, double* __restrict__ pv)
{
    __shared__ __align__(16) double s_w[4][kFoldStep];
    const int lane = threadIdx.x & 31;
    const int64_t nr = *nruns;
    for (int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; r < nr;
         r += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const longlong2 run = runs[r];
        const int64_t v = (int64_t)(keys[run.x] >> lb);
        const double x = fold_run<true>(ws + run.x, run.y - run.x, pv[v], s_w[threadIdx.x >> 5]);
        if (lane == 0) pv[v] = x;
    }
}

template <int NW, int G, int W, bool kOne>
int launch_rounds(rtr_graph* g, const RoundArgs& ra, int64_t units, cudaStream_t st)
{
    if (units == 0) return RTR_OK;
    const size_t smem = sizeof(WinSmem<NW, G, W>);
    RTR_CUDA_TRY(cudaFuncSetAttribute(k_clean_rounds<NW, G, W, kOne>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    k_clean_rounds<NW, G, W, kOne><<<(unsigned)units, 32 * NW, smem, st>>>(ra);
    g->launches += 1;
    RTR_CUDA_TRY(cudaGetLastError());
    return RTR_OK;
}

}  // namespace

// A log of up to this size is simply asked for (the device's free memory takes 64 us
// to learn); a larger one must leave this much of it to others.
constexpr int64_t kLogSmall = 256ll << 20;
constexpr int64_t kLogMargin = 1ll << 30;

bool clean_rounds_reserve(rtr_graph* g, Scratch& sc, int64_t stack_entries, int64_t log_entries, RoundReplay* rr)
{
    const int64_t pops = stack_entries, logs = log_entries, cnt = 3 * logs;
    const size_t sizes[] = {sizeof(PopLog) * ((size_t)pops + 1),
                            (size_t)g->tl_len + 16,
                            sizeof(uint32_t) * ((size_t)pops + 1),
                            sizeof(uint32_t) * ((size_t)pops + 1),
                            sizeof(uint32_t) * (size_t)scan_temp_elems(pops + 1),
                            sizeof(double) * ((size_t)logs + 1),
                            sizeof(uint64_t) * ((size_t)cnt + 1),
                            sizeof(uint64_t) * ((size_t)cnt + 1),
                            radix_temp_bytes(cnt),
                            sizeof(double) * ((size_t)cnt + 1),
                            sizeof(longlong2) * ((size_t)(cnt / kLongRun) + 2),
                            sizeof(unsigned) * 2};
    constexpr int kParts = sizeof sizes / sizeof sizes[0];
    int64_t need = 0;
    for (const size_t b : sizes) need += (int64_t)b;
    if (g->clean_log_limit >= 0 && need > g->clean_log_limit) return false;
    if (need > kLogSmall && need + kLogMargin > (int64_t)device_avail_bytes(g)) return false;
    void* part[kParts];
    for (int k = 0; k < kParts; ++k)
        if (!(part[k] = sc.get(sizes[k]))) {
            cudaGetLastError();  // the units replay without the log
            return false;
        }
    rr->pops_cap = pops;
    rr->logs_cap = logs;
    rr->plog = (PopLog*)part[0];
    rr->live8 = (uint8_t*)part[1];
    rr->pcnt = (uint32_t*)part[2];
    rr->poff = (uint32_t*)part[3];
    rr->ptmp = (uint32_t*)part[4];
    rr->wlog = (double*)part[5];
    rr->keys = (uint64_t*)part[6];
    rr->alt = (uint64_t*)part[7];
    rr->rtmp = part[8];
    rr->ws = (double*)part[9];
    rr->runs = (longlong2*)part[10];
    rr->nruns = (unsigned*)part[11];
    return true;
}

int clean_rounds_launch(rtr_graph* g, const cudaStream_t* st, EdgeRec* rec, const StackEntry* seeds,
                        const UnitDesc* units, const uint64_t* order, const int64_t* kinds, StackEntry* stacks,
                        RoundReplay* rr)
{
    rr->rec = rec;
    cudaStream_t s = g->stream;
    RTR_CUDA_TRY(cudaMemsetAsync(rr->plog, 0xff, sizeof(PopLog) * ((size_t)rr->pops_cap + 1), s));
    RTR_CUDA_TRY(cudaMemsetAsync(rr->live8, 0, (size_t)g->tl_len + 16, s));
    // the replays on side streams run after everything above
    cudaEvent_t ready = nullptr;
    for (int k = 0; k < UNIT_WARP; ++k) {
        if (kinds[k] == 0 || st[k] == s) continue;
        if (!ready) {
            RTR_CUDA_TRY(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
            cudaEventRecord(ready, s);
        }
        cudaStreamWaitEvent(st[k], ready, 0);
    }
    if (ready) cudaEventDestroy(ready);
    RoundArgs ra{g->tl,    rec,       1 / (double)g->n,         seeds,  units,     order, stacks,
                 rr->plog, rr->live8, (unsigned*)(g->ctr + 1), g->ctr, g->ctr + 2};
    RTR_TRY((launch_rounds<8, 0, 8, false>(g, ra, kinds[UNIT_WIDE], st[UNIT_WIDE])));
    ra.order += kinds[UNIT_WIDE];
    RTR_TRY((launch_rounds<8, 0, 8, true>(g, ra, kinds[UNIT_WIDE_FEW], st[UNIT_WIDE_FEW])));
    ra.order += kinds[UNIT_WIDE_FEW];
    RTR_TRY((launch_rounds<8, 16, 16, false>(g, ra, kinds[UNIT_NARROW], st[UNIT_NARROW])));
    ra.order += kinds[UNIT_NARROW];
    return launch_rounds<8, 16, 16, true>(g, ra, kinds[UNIT_NARROW_FEW], st[UNIT_NARROW_FEW]);
}

int clean_rounds_finish(rtr_graph* g, RoundReplay* rr)
{
    cudaStream_t s = g->stream;
    const int64_t pops = rr->pops_cap, logs = rr->logs_cap, cnt = 3 * logs;
    if (logs == 0) return RTR_OK;
    const int lb = bits_for((uint64_t)logs);
    const int vb = bits_for((uint64_t)g->n);
    RTR_CUDA_TRY(cudaMemsetAsync(rr->nruns, 0, sizeof(unsigned) * 2, s));
    // an unused key keeps a vertex past the last
    RTR_CUDA_TRY(cudaMemsetAsync(rr->keys, 0xff, sizeof(uint64_t) * (size_t)cnt, s));
    k_pop_counts<<<grid_for(pops, kBlock), kBlock, 0, s>>>(rr->plog, pops, rr->pcnt);
    RTR_TRY(exclusive_scan_u32(rr->pcnt, rr->poff, pops, nullptr, rr->ptmp, s));
    k_log_keys<<<grid_for(8 * pops, kBlock), kBlock, 0, s>>>(rr->rec, rr->plog, rr->poff, pops, g->tl, rr->live8,
                                                             g->fwd, g->esrc, g->nbors, 1 / (double)g->n, lb,
                                                             rr->keys, rr->wlog, (unsigned*)(g->ctr + 1), g->ctr + 2);
    // the keys come in log order, so a stable sort on the vertex bits suffices
    uint64_t* sorted = nullptr;
    RTR_TRY(radix_sort_bits_u64(rr->keys, rr->alt, cnt, lb, lb + vb, rr->rtmp, s, &sorted));
    k_log_gather<<<grid_for(cnt, kBlock), kBlock, 0, s>>>(sorted, cnt, g->n, lb, rr->wlog, rr->ws, g->pv, rr->runs,
                                                          rr->nruns);
    k_fold_long_runs<<<grid_for(1ll << 40, 128, 8), 128, 0, s>>>(rr->runs, rr->nruns, sorted, lb, rr->ws, g->pv);
    g->launches += 4 + take_primitive_launches();
    RTR_CUDA_TRY(cudaGetLastError());
    return RTR_OK;
}

}  // namespace rtr
