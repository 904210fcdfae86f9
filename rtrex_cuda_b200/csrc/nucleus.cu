// The nucleus (truss-hierarchy) path on the device, bit-exact to the
// reference's nucleus driver (RTRex_Sequential/clustering/nucleus.cpp:12-81):
//
//   1. relabel by (degree, id)      CGraph::renameByDegreeOrderMapping (Graph.cpp:261-310):
//                                   a radix sort of (degree, id) keys, then the CSR of the
//                                   relabelled pairs built like any graph (rows ascending)
//   2. per-edge triangle lists      storeAllTriangles (Escape/Nucleus.h:125-163): the list
//                                   layout of count_triangles on the relabelled graph -- for
//                                   each forward edge (i, j), i < j, its common neighbours
//                                   ascending, with the forward ranks of (i, k) and (j, k)
//   3. integer peel                nuclei's deletion loop (Nucleus.h:349-458).  A cascade stays
//                                   among edges connected by triangles, so each such unit replays
//                                   its own deletions, one warp per unit, in the reference's order:
//                                   per threshold c, the unit's edges with fewer than c live
//                                   triangles pushed in slot order, popped last-first, each pop's
//                                   triangles taken 32 at a time (within one pop they touch
//                                   distinct edges; pushes are appended in triangle order).  The
//                                   reference's stack holds all units' seeds of a level in slot
//                                   order, so its deletion order is (c, seed descending, order
//                                   within the unit): two stable sorts
//   4. edge hierarchy and clusters  findConnectedComponent / completeCluster (Nucleus.h:169-301,
//                                   :460-563) by union-find, level by level from the top.  The
//                                   reference joins two edges of a triangle at the smaller of
//                                   their kappas; a component that gains edges at a level becomes
//                                   a cluster there, the next clusters inside it its children.
//                                   Its root in the reference is the last walk started in it, and
//                                   a walk starts at an edge iff no triangle neighbour of the same
//                                   kappa was deleted before it (such a neighbour's walk reaches
//                                   it); clusters of a level come in the roots' deletion order.
//                                   Members are the new edges' endpoints and the children's
//                                   members, made distinct and ascending by a radix sort (the
//                                   std::set order of relabelled ids), then mapped back to the
//                                   original labels.
//
// Measured (B200, 30,011-edge block model): one warp's peel of the whole graph took
// 27.8 ms and one thread's walk of the hierarchy 31.9 ms; the whole call takes 1.8 ms
// now (largest unit 305 edges).  A graph that is one unit still peels in one warp:
// a 40,000-edge R-MAT graph 84 ms.
//
// Edges are identified by forward rank of the relabelled CSR (the reference uses
// the forward slot; both are ordered the same way and only compared for equality
// past the seeding).  No floating point is involved.
#include "../../include/rtr.h"
#include "primitives.cuh"
#include "rtr_graph.cuh"
#include "unionfind.cuh"

#include <algorithm>
#include <cstdio>
#include <string>
#include <vector>

namespace rtr {
int make_graph_handle(int64_t n, int device, rtr_graph** out);
}

using namespace rtr;

namespace {

constexpr int kBlock = 256;

__global__ void k_nuc_keys(const int32_t* __restrict__ deg, int64_t n, int B, uint64_t* __restrict__ keys)
{
    for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x)
        keys[v] = ((uint64_t)deg[v] << B) | (uint64_t)v;
}

__global__ void k_nuc_rank(const uint64_t* __restrict__ sorted, int64_t n, uint64_t mask, int32_t* __restrict__ inv,
                           int32_t* __restrict__ newid)
{
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
        const int32_t v = (int32_t)(sorted[r] & mask);
        inv[r] = v;
        newid[v] = (int32_t)r;
    }
}

__global__ void k_nuc_pairs(const int32_t* __restrict__ fwd, const int32_t* __restrict__ esrc,
                            const int32_t* __restrict__ nb, const int32_t* __restrict__ newid, int64_t m,
                            int64_t* __restrict__ u, int64_t* __restrict__ v)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
        const int32_t f = fwd[k];
        u[k] = newid[esrc[f]];
        v[k] = newid[nb[f]];
    }
}

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ int warp_excl(int x, int lane, int* total)
{
    int incl = x;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
    }
    *total = __shfl_sync(kFull, incl, 31);
    return incl - x;
}

constexpr unsigned NUC_ERR_STACK = 4;

// Edges by forward rank: live triangles, and the level (-1: not deleted yet; an
// edge without triangles has kappa 0 and takes no further part).
__global__ void k_nuc_init(const int32_t* __restrict__ fwd, const uint32_t* __restrict__ sup, int64_t m,
                           int32_t* __restrict__ tc, int32_t* __restrict__ kappa, int32_t* __restrict__ root,
                           uint32_t* __restrict__ carries)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
        const uint32_t s = sup[fwd[k]];
        tc[k] = (int32_t)s;
        kappa[k] = s ? -1 : 0;
        root[k] = (int32_t)k;
        carries[k] = s ? 1u : 0u;
    }
}

// Units: edges joined by the triangles (each taken from its smallest edge's list).
__global__ void k_nuc_unite(const int32_t* __restrict__ fwd, const int32_t* __restrict__ nb,
                            const int64_t* __restrict__ tl_off, const TriEntry* __restrict__ tl, int64_t m,
                            int32_t* __restrict__ root)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x) {
        const int32_t f = fwd[k], b = nb[f];
        for (int64_t t = tl_off[f]; t < tl_off[f + 1]; ++t) {
            const TriEntry te = tl[t];
            if (te.z < b) continue;
            uf_unite(root, (int32_t)k, te.raz);
            uf_unite(root, (int32_t)k, te.rbz);
        }
    }
}

__global__ void k_nuc_iota(int32_t* __restrict__ p, int64_t m)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x)
        p[k] = (int32_t)k;
}

__global__ void k_nuc_unit_keys(const uint32_t* __restrict__ carries, const uint32_t* __restrict__ pos, int64_t m,
                                int rb, int32_t* __restrict__ root, uint64_t* __restrict__ keys)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < m; k += (int64_t)gridDim.x * blockDim.x)
        if (carries[k]) keys[pos[k]] = ((uint64_t)uf_find(root, (int32_t)k) << rb) | (uint64_t)k;
}

__global__ void k_nuc_unit_list(const uint64_t* __restrict__ sorted, int64_t mc, int rb, const int32_t* __restrict__ tc,
                                int32_t* __restrict__ list, int64_t* __restrict__ sup, uint32_t* __restrict__ head)
{
    const uint64_t mask = (1ull << rb) - 1;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < mc; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t k = sorted[i];
        list[i] = (int32_t)(k & mask);
        sup[i] = tc[k & mask];
        head[i] = i == 0 || (sorted[i - 1] >> rb) != (k >> rb) ? 1u : 0u;
    }
}

__global__ void k_nuc_unit_begin(const uint32_t* __restrict__ head, const uint32_t* __restrict__ hpos, int64_t mc,
                                 int64_t* __restrict__ ub)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < mc; i += (int64_t)gridDim.x * blockDim.x)
        if (head[i]) ub[hpos[i]] = i;
}

// Largest units first.
__global__ void k_nuc_unit_order(const int64_t* __restrict__ ub, int64_t nu, int64_t mc, uint64_t* __restrict__ keys)
{
    for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < nu; u += (int64_t)gridDim.x * blockDim.x) {
        const int64_t size = (u + 1 < nu ? ub[u + 1] : mc) - ub[u];
        keys[u] = ((0x7fffffffull - (uint64_t)size) << 32) | (uint64_t)u;
    }
}

struct PeelArgs {
    const int32_t* fwd;       // rank -> forward slot
    const int64_t* tl_off;    // slot -> first triangle entry
    const TriEntry* tl;
    int32_t* tc;              // rank -> live triangles
    int32_t* kappa;           // rank -> level - 1 at deletion
    const int32_t* list;      // the units' edges, ascending within a unit
    const int64_t* ub;        // unit -> first in list
    const int64_t* psup;      // list position -> triangle counts before it
    const uint64_t* order;    // units by size
    int64_t nu, mc;
    int32_t* stack;           // unit u's region: ub[u] + 2/3 psup[ub[u]] + 64 u
    // the deletions of each unit, in its order, from list position ub[u]
    int32_t* del_edge;
    int32_t* del_seed;        // the seed whose cascade it is
    int32_t* del_level;       // c
    unsigned* next;           // [0] unit queue, [1] highest c, [2] error bits
};

__global__ void __launch_bounds__(128) k_nuc_peel(PeelArgs a)
{
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    while (true) {
        unsigned q = 0;
        if (lane == 0) q = atomicAdd(&a.next[0], 1u);
        q = __shfl_sync(kFull, q, 0);
        if ((int64_t)q >= a.nu) return;
        const int64_t u = (int64_t)(uint32_t)a.order[q];
        const int64_t b = a.ub[u], e = u + 1 < a.nu ? a.ub[u + 1] : a.mc;
        int32_t* stack = a.stack + b + 2 * a.psup[b] / 3 + 64 * u;
        const int64_t cap = (e - b) + 2 * (a.psup[e] - a.psup[b]) / 3 + 64;
        int64_t done = 0;
        int c = 0;
        bool err = false;
        while (done < e - b && !err) {
            // the next level that has seeds, and its seeds in slot order
            int least = INT32_MAX;
            for (int64_t i = b + lane; i < e; i += 32) {
                const int32_t k = a.list[i];
                if (a.kappa[k] < 0) least = min(least, a.tc[k]);
            }
            least = __reduce_min_sync(kFull, least);
            c = max(c, least) + 1;
            int64_t top = 0;
            for (int64_t i0 = b; i0 < e; i0 += 32) {
                int32_t k = 0;
                bool push = false;
                if (i0 + lane < e) {
                    k = a.list[i0 + lane];
                    push = a.kappa[k] < 0 && a.tc[k] < c;
                }
                const unsigned pm = __ballot_sync(kFull, push);
                if (push) stack[top + __popc(pm & lt)] = k;
                top += __popc(pm);
            }
            int64_t seeds = top;  // stack[0, seeds): seeds not popped yet
            int32_t seed = 0;
            __syncwarp();
            while (top > 0 && !err) {
                const int32_t x = stack[--top];
                if (top < seeds) {
                    seeds = top;
                    seed = x;
                }
                const bool gone = a.kappa[x] >= 0;
                __syncwarp();
                if (gone) continue;
                if (lane == 0) {
                    a.kappa[x] = c - 1;
                    a.del_edge[b + done] = x;
                    a.del_seed[b + done] = seed;
                    a.del_level[b + done] = c;
                }
                ++done;
                __syncwarp();
                const int32_t f = a.fwd[x];
                const int64_t t1 = a.tl_off[f + 1];
                for (int64_t tb = a.tl_off[f]; tb < t1; tb += 32) {
                    int32_t ra = 0, rb = 0;
                    bool live = false;
                    if (tb + lane < t1) {
                        const TriEntry te = a.tl[tb + lane];
                        ra = te.raz;  // (i, k)
                        rb = te.rbz;  // (j, k)
                        live = a.kappa[ra] < 0 && a.kappa[rb] < 0;
                    }
                    bool p1 = false, p2 = false;
                    if (live) {  // the triangle dies: both other edges lose one
                        p1 = --a.tc[ra] < c;
                        p2 = --a.tc[rb] < c;
                    }
                    int tp = 0;
                    const int op = warp_excl((p1 ? 1 : 0) + (p2 ? 1 : 0), lane, &tp);
                    if (top + tp > cap) {
                        err = true;
                        break;
                    }
                    if (p1) stack[top + op] = ra;
                    if (p2) stack[top + op + (p1 ? 1 : 0)] = rb;
                    top += tp;
                    __syncwarp();
                }
            }
        }
        if (lane == 0) {
            atomicMax(&a.next[1], (unsigned)c);
            if (err) atomicOr(&a.next[2], (unsigned)NUC_ERR_STACK);
        }
    }
}

// The deletion order: by seed (highest first), then by level, both stable over
// the units' own orders.
__global__ void k_nuc_seed_keys(const int32_t* __restrict__ del_seed, int64_t mc, int64_t m, int pb,
                                uint64_t* __restrict__ keys)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < mc; i += (int64_t)gridDim.x * blockDim.x)
        keys[i] = ((uint64_t)(m - 1 - del_seed[i]) << pb) | (uint64_t)i;
}

__global__ void k_nuc_level_keys(uint64_t* __restrict__ keys, int64_t mc, int pb, const int32_t* __restrict__ del_level,
                                 unsigned* __restrict__ hist)
{
    const uint64_t mask = (1ull << pb) - 1;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < mc; i += (int64_t)gridDim.x * blockDim.x) {
        const uint64_t p = keys[i] & mask;
        const int32_t c = del_level[p];
        keys[i] = ((uint64_t)c << pb) | p;
        atomicAdd(&hist[c], 1u);
    }
}

__global__ void k_nuc_deletions(const uint64_t* __restrict__ keys, int64_t mc, int pb,
                                const int32_t* __restrict__ del_edge, int32_t* __restrict__ ord,
                                int32_t* __restrict__ dtime)
{
    const uint64_t mask = (1ull << pb) - 1;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < mc; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t e = del_edge[keys[i] & mask];
        ord[i] = e;
        dtime[e] = (int32_t)i;
    }
}

struct LevelArgs {
    const int32_t* fwd;
    const int32_t* esrc;
    const int32_t* nb;
    const int64_t* tl_off;
    const TriEntry* tl;
    const int32_t* kappa;
    const int32_t* dtime;
    const int32_t* ord;      // the level's edges, in deletion order
    int64_t cnt;
    int32_t lv;
    int32_t* comp;           // union-find over edges, for the levels so far
    int32_t* croot;          // [cnt] the edges' components
    uint32_t* is_start;      // [cnt]
    int32_t* best;           // component -> last start of this level (-1)
    uint32_t* ecount;        // component -> its edges of this level
    int32_t* clid;           // component -> its newest cluster
    int32_t* clstamp;        // component -> the level of that cluster
};

// Join the level's edges with their triangle neighbours of at least its kappa;
// an edge starts a walk iff none of the same kappa was deleted before it.
__global__ void k_nuc_join(LevelArgs a)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.cnt; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t x = a.ord[i], f = a.fwd[x];
        const int32_t dx = a.dtime[x];
        bool start = true;
        for (int64_t t = a.tl_off[f]; t < a.tl_off[f + 1]; ++t) {
            const TriEntry te = a.tl[t];
            const int32_t y[2] = {te.raz, te.rbz};
            for (int q = 0; q < 2; ++q) {
                const int32_t k = a.kappa[y[q]];
                if (k < a.lv) continue;
                uf_unite(a.comp, x, y[q]);
                if (k == a.lv && a.dtime[y[q]] < dx) start = false;
            }
        }
        a.is_start[i] = start ? 1u : 0u;
    }
}

__global__ void k_nuc_comps(LevelArgs a)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.cnt; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t x = a.ord[i];
        const int32_t r = uf_find(a.comp, x);
        a.croot[i] = r;
        atomicAdd(&a.ecount[r], 1u);
        if (a.is_start[i]) atomicMax(&a.best[r], a.dtime[x]);
    }
}

// is_start becomes: the root of its component's cluster.
__global__ void k_nuc_roots(LevelArgs a)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.cnt; i += (int64_t)gridDim.x * blockDim.x)
        a.is_start[i] = a.best[a.croot[i]] == a.dtime[a.ord[i]] ? 1u : 0u;
}

struct Clusters {
    int64_t* c;
    int64_t* nv;
    int64_t* ne;
    int64_t* parent;
    int64_t* voff;  // first member
    int32_t* rep;   // one of its edges
};

__global__ void k_nuc_clusters(LevelArgs a, const uint32_t* __restrict__ pos, int64_t ncl, Clusters cl)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.cnt; i += (int64_t)gridDim.x * blockDim.x) {
        if (!a.is_start[i]) continue;
        const int32_t r = a.croot[i];
        const int64_t k = ncl + pos[i];
        cl.c[k] = a.lv;
        cl.ne[k] = a.ecount[r];
        cl.parent[k] = -1;
        cl.rep[k] = a.ord[i];
        a.clid[r] = (int32_t)k;
        a.clstamp[r] = a.lv;
        a.best[r] = -1;
        a.ecount[r] = 0;
    }
}

// The clusters that this level's components take in: their parents, and how many
// members they bring.
__global__ void k_nuc_children(LevelArgs a, int64_t ncl, Clusters cl, int64_t* __restrict__ brings)
{
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < ncl; k += (int64_t)gridDim.x * blockDim.x) {
        brings[k] = 0;
        if (cl.parent[k] >= 0) continue;
        const int32_t r = uf_find(a.comp, cl.rep[k]);
        if (a.clstamp[r] != a.lv) continue;
        const int32_t p = a.clid[r];
        cl.parent[k] = p;
        atomicAdd((unsigned long long*)&cl.ne[p], (unsigned long long)cl.ne[k]);
        brings[k] = cl.nv[k];
    }
}

// Member keys (cluster - first of the level, vertex): the edges' endpoints, then the children's members.
__global__ void k_nuc_edge_members(LevelArgs a, int64_t ncl, int B, uint64_t* __restrict__ keys)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.cnt; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t f = a.fwd[a.ord[i]];
        const uint64_t k = (uint64_t)(a.clid[a.croot[i]] - ncl) << B;
        keys[2 * i] = k | (uint64_t)a.esrc[f];
        keys[2 * i + 1] = k | (uint64_t)a.nb[f];
    }
}

__global__ void k_nuc_child_members(int64_t ncl, Clusters cl, const int64_t* __restrict__ brings,
                                    const int64_t* __restrict__ at, const int32_t* __restrict__ vert, int B,
                                    uint64_t* __restrict__ keys)
{
    const int lane = threadIdx.x & 31;
    for (int64_t k = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; k < ncl;
         k += ((int64_t)gridDim.x * blockDim.x) >> 5) {
        const int64_t n = brings[k];
        const uint64_t p = (uint64_t)(cl.parent[k] - ncl) << B;
        for (int64_t j = lane; j < n; j += 32) keys[at[k] + j] = p | (uint64_t)vert[cl.voff[k] + j];
    }
}

__global__ void k_nuc_distinct(const uint64_t* __restrict__ keys, int64_t cnt, uint32_t* __restrict__ flag)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x)
        flag[i] = i == 0 || keys[i - 1] != keys[i] ? 1u : 0u;
}

__global__ void k_nuc_members(const uint64_t* __restrict__ keys, int64_t cnt, const uint32_t* __restrict__ flag,
                              const uint32_t* __restrict__ pos, const unsigned* __restrict__ distinct, int64_t ncl,
                              int B, int64_t vbase, Clusters cl, int32_t* __restrict__ vert)
{
    const uint64_t mask = (1ull << B) - 1;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < cnt; i += (int64_t)gridDim.x * blockDim.x) {
        if (flag[i]) vert[vbase + pos[i]] = (int32_t)(keys[i] & mask);
        const int64_t k = ncl + (int64_t)(keys[i] >> B);
        if (i == 0 || (keys[i - 1] >> B) != (keys[i] >> B)) cl.voff[k] = vbase + pos[i];
        // the cluster's last key: one past its last member (nv is completed by k_nuc_sizes)
        if (i + 1 == cnt || (keys[i + 1] >> B) != (keys[i] >> B))
            cl.nv[k] = vbase + (i + 1 == cnt ? (int64_t)*distinct : (int64_t)pos[i + 1]);
    }
}

__global__ void k_nuc_sizes(int64_t from, int64_t to, Clusters cl)
{
    for (int64_t k = from + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < to; k += (int64_t)gridDim.x * blockDim.x)
        cl.nv[k] -= cl.voff[k];
}

__global__ void k_nuc_labels(const int32_t* __restrict__ vert, int64_t cnt, const int32_t* __restrict__ inv,
                             int64_t* __restrict__ out)
{
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < cnt; p += (int64_t)gridDim.x * blockDim.x)
        out[p] = inv[vert[p]];
}

// The relabelled graph, whose launches are its owner's.
struct GraphGuard {
    rtr_graph* owner;
    rtr_graph* g = nullptr;
    ~GraphGuard()
    {
        if (!g) return;
        owner->launches += g->launches;
        rtr_graph_destroy(g);
    }
};

int nucleus_run(rtr_graph* g)
{
    take_primitive_launches();  // what a call that failed left uncounted is not this one's
    const int64_t n = g->n, m = g->m;
    cudaStream_t s = g->stream;
    g->nuc_done = false;
    g->nuc_c.clear();
    g->nuc_nv.clear();
    g->nuc_ne.clear();
    g->nuc_parent.clear();
    g->nuc_off.assign(1, 0);
    g->nuc_vert.clear();
    if (m == 0) {  // no edges, no levels, no clusters
        g->nuc_done = true;
        return RTR_OK;
    }
    const int B = bits_for((uint64_t)(n - 1));
    const uint64_t mask = (1ull << B) - 1;
    Scratch isc(g);
    GraphGuard rel{g};
    int32_t* inv = (int32_t*)isc.get(sizeof(int32_t) * (n + 1));
    {
        Scratch sc(g);
        uint64_t* k1 = (uint64_t*)sc.get(sizeof(uint64_t) * (n + 1));
        uint64_t* k2 = (uint64_t*)sc.get(sizeof(uint64_t) * (n + 1));
        void* rtmp = sc.get(radix_temp_bytes(n));
        int32_t* newid = (int32_t*)sc.get(sizeof(int32_t) * (n + 1));
        int64_t* du = (int64_t*)sc.get(sizeof(int64_t) * (m + 1));
        int64_t* dv = (int64_t*)sc.get(sizeof(int64_t) * (m + 1));
        if (!k1 || !k2 || !rtmp || !newid || !du || !dv || !inv) {
            set_error("device allocation failed (nucleus relabel)");
            return RTR_ERR_CUDA;
        }
        const int gn = grid_for(n, kBlock);
        k_nuc_keys<<<gn, kBlock, 0, s>>>(g->deg, n, B, k1);
        uint64_t* sorted = nullptr;
        RTR_TRY(radix_sort_u64(k1, k2, n, B + bits_for((uint64_t)g->m2), rtmp, s, &sorted));
        k_nuc_rank<<<gn, kBlock, 0, s>>>(sorted, n, mask, inv, newid);
        k_nuc_pairs<<<grid_for(m, kBlock), kBlock, 0, s>>>(g->fwd, g->esrc, g->nbors, newid, m, du, dv);
        g->launches += 3 + take_primitive_launches();
        RTR_CUDA_TRY(cudaGetLastError());
        RTR_CUDA_TRY(cudaStreamSynchronize(s));
        int rc = make_graph_handle(n, g->device, &rel.g);
        if (rc) return rc;
        rc = build_csr(rel.g, du, dv, m, false);
        if (!rc) RTR_CUDA_TRY(cudaStreamSynchronize(rel.g->stream));
        if (rc) return rc;
    }
    rtr_graph* r = rel.g;
    r->count_mode = 1;  // the lists are the reference's triangle lists
    int rc = count_triangles(r);
    if (rc) return rc;
    cudaStream_t rs = r->stream;
    Scratch sc(r);
    const int gm = grid_for(m, kBlock);
    const int rb = bits_for((uint64_t)m);
    auto failed = [](const char* what) {
        set_error("device allocation failed (nucleus %s)", what);
        return RTR_ERR_CUDA;
    };
    // ---- the peel's units
    int32_t* tc = (int32_t*)sc.get(sizeof(int32_t) * (m + 1));
    int32_t* kappa = (int32_t*)sc.get(sizeof(int32_t) * (m + 1));
    int32_t* comp = (int32_t*)sc.get(sizeof(int32_t) * (m + 1));
    uint32_t* carries = (uint32_t*)sc.get(sizeof(uint32_t) * (m + 1));
    uint32_t* cpos = (uint32_t*)sc.get(sizeof(uint32_t) * (m + 1));
    uint32_t* stmp = (uint32_t*)sc.get(sizeof(uint32_t) * scan_temp_elems(m + 1));
    unsigned* next = (unsigned*)sc.get(sizeof(unsigned) * 8);
    if (!tc || !kappa || !comp || !carries || !cpos || !stmp || !next) return failed("edges");
    RTR_CUDA_TRY(cudaMemsetAsync(next, 0, sizeof(unsigned) * 8, rs));
    k_nuc_init<<<gm, kBlock, 0, rs>>>(r->fwd, r->sup, m, tc, kappa, comp, carries);
    RTR_TRY(exclusive_scan_u32(carries, cpos, m, next + 4, stmp, rs));
    k_nuc_unite<<<gm, kBlock, 0, rs>>>(r->fwd, r->nbors, r->tl_off, r->tl, m, comp);
    g->launches += 2 + take_primitive_launches();
    unsigned mc32 = 0;
    RTR_CUDA_TRY(cudaGetLastError());
    RTR_CUDA_TRY(cudaMemcpyAsync(&mc32, next + 4, sizeof mc32, cudaMemcpyDeviceToHost, rs));
    RTR_CUDA_TRY(cudaStreamSynchronize(rs));
    const int64_t mc = mc32;  // edges with triangles
    if (mc == 0) {
        g->nuc_done = true;
        return RTR_OK;
    }
    const int gc = grid_for(mc, kBlock), pb = bits_for((uint64_t)mc);
    uint64_t* k1 = (uint64_t*)sc.get(sizeof(uint64_t) * (mc + 1));
    uint64_t* k2 = (uint64_t*)sc.get(sizeof(uint64_t) * (mc + 1));
    void* rtmp = sc.get(radix_temp_bytes(mc));
    int32_t* list = (int32_t*)sc.get(sizeof(int32_t) * (mc + 1));
    int64_t* lsup = (int64_t*)sc.get(sizeof(int64_t) * (mc + 1));
    int64_t* psup = (int64_t*)sc.get(sizeof(int64_t) * (mc + 2));
    uint32_t* head = (uint32_t*)sc.get(sizeof(uint32_t) * (mc + 1));
    uint32_t* hpos = (uint32_t*)sc.get(sizeof(uint32_t) * (mc + 1));
    int64_t* ub = (int64_t*)sc.get(sizeof(int64_t) * (mc + 1));
    int64_t* ltmp = (int64_t*)sc.get(sizeof(int64_t) * scan_temp_elems(mc + 1));
    if (!k1 || !k2 || !rtmp || !list || !lsup || !psup || !head || !hpos || !ub || !ltmp) return failed("units");
    k_nuc_unit_keys<<<gm, kBlock, 0, rs>>>(carries, cpos, m, rb, comp, k1);
    uint64_t* by_unit = nullptr;
    RTR_TRY(radix_sort_u64(k1, k2, mc, 2 * rb, rtmp, rs, &by_unit));
    k_nuc_unit_list<<<gc, kBlock, 0, rs>>>(by_unit, mc, rb, tc, list, lsup, head);
    RTR_TRY(exclusive_scan_i64(lsup, psup, mc, psup + mc, ltmp, rs));
    RTR_TRY(exclusive_scan_u32(head, hpos, mc, next + 5, stmp, rs));
    k_nuc_unit_begin<<<gc, kBlock, 0, rs>>>(head, hpos, mc, ub);
    unsigned nu32 = 0;
    RTR_CUDA_TRY(cudaGetLastError());
    RTR_CUDA_TRY(cudaMemcpyAsync(&nu32, next + 5, sizeof nu32, cudaMemcpyDeviceToHost, rs));
    RTR_CUDA_TRY(cudaStreamSynchronize(rs));
    const int64_t nu = nu32;
    uint64_t* o1 = (uint64_t*)sc.get(sizeof(uint64_t) * (nu + 1));
    uint64_t* o2 = (uint64_t*)sc.get(sizeof(uint64_t) * (nu + 1));
    void* otmp = sc.get(radix_temp_bytes(nu));
    PeelArgs pa;
    pa.fwd = r->fwd;
    pa.tl_off = r->tl_off;
    pa.tl = r->tl;
    pa.tc = tc;
    pa.kappa = kappa;
    pa.list = list;
    pa.ub = ub;
    pa.psup = psup;
    pa.nu = nu;
    pa.mc = mc;
    pa.stack = (int32_t*)sc.get(sizeof(int32_t) * (size_t)(mc + 2 * (r->tl_len / 3) + 64 * nu + 64));
    pa.del_edge = (int32_t*)sc.get(sizeof(int32_t) * (mc + 1));
    pa.del_seed = (int32_t*)sc.get(sizeof(int32_t) * (mc + 1));
    pa.del_level = (int32_t*)sc.get(sizeof(int32_t) * (mc + 1));
    pa.next = next;
    if (!o1 || !o2 || !otmp || !pa.stack || !pa.del_edge || !pa.del_seed || !pa.del_level) return failed("peel");
    k_nuc_unit_order<<<grid_for(nu, kBlock), kBlock, 0, rs>>>(ub, nu, mc, o1);
    uint64_t* by_size = nullptr;
    RTR_TRY(radix_sort_bits_u64(o1, o2, nu, 32, 64, otmp, rs, &by_size));
    pa.order = by_size;
    // the largest unit's chain bounds the peel
    k_nuc_peel<<<(int)std::min<int64_t>((nu + 3) / 4, grid_for(1ll << 40, 128, 16)), 128, 0, rs>>>(pa);
    // the deletion order
    k_nuc_seed_keys<<<gc, kBlock, 0, rs>>>(pa.del_seed, mc, m, pb, k1);
    uint64_t* seq = nullptr;
    RTR_TRY(radix_sort_bits_u64(k1, k2, mc, pb, pb + rb, rtmp, rs, &seq));
    g->launches += 6 + take_primitive_launches();
    unsigned pk[3] = {0, 0, 0};
    RTR_CUDA_TRY(cudaGetLastError());
    RTR_CUDA_TRY(cudaMemcpyAsync(pk, next, sizeof pk, cudaMemcpyDeviceToHost, rs));
    RTR_CUDA_TRY(cudaStreamSynchronize(rs));
    if (pk[2]) {
        set_error("nucleus peel reported 0x%x", pk[2]);
        return RTR_ERR_DEVICE;
    }
    const int64_t max_c = pk[1];
    unsigned* hist = (unsigned*)sc.get(sizeof(unsigned) * (max_c + 2));
    int32_t* ord = (int32_t*)sc.get(sizeof(int32_t) * (mc + 1));
    int32_t* dtime = (int32_t*)sc.get(sizeof(int32_t) * (m + 1));
    if (!hist || !ord || !dtime) return failed("order");
    RTR_CUDA_TRY(cudaMemsetAsync(hist, 0, sizeof(unsigned) * (max_c + 2), rs));
    k_nuc_level_keys<<<gc, kBlock, 0, rs>>>(seq, mc, pb, pa.del_level, hist);
    RTR_TRY(radix_sort_bits_u64(seq, seq == k1 ? k2 : k1, mc, pb, pb + bits_for((uint64_t)max_c), rtmp, rs, &seq));
    k_nuc_deletions<<<gc, kBlock, 0, rs>>>(seq, mc, pb, pa.del_edge, ord, dtime);
    std::vector<unsigned> per_level((size_t)max_c + 2);
    RTR_CUDA_TRY(cudaMemcpyAsync(per_level.data(), hist, sizeof(unsigned) * (max_c + 2), cudaMemcpyDeviceToHost, rs));
    // ---- the hierarchy, from the highest level down
    LevelArgs la;
    la.fwd = r->fwd;
    la.esrc = r->esrc;
    la.nb = r->nbors;
    la.tl_off = r->tl_off;
    la.tl = r->tl;
    la.kappa = kappa;
    la.dtime = dtime;
    la.comp = comp;
    la.croot = (int32_t*)sc.get(sizeof(int32_t) * (mc + 1));
    la.is_start = carries;  // free by now
    la.best = (int32_t*)sc.get(sizeof(int32_t) * (m + 1));
    la.ecount = (uint32_t*)sc.get(sizeof(uint32_t) * (m + 1));
    la.clid = (int32_t*)sc.get(sizeof(int32_t) * (m + 1));
    la.clstamp = (int32_t*)sc.get(sizeof(int32_t) * (m + 1));
    Clusters cl;
    cl.c = (int64_t*)sc.get(sizeof(int64_t) * (mc + 1));
    cl.nv = (int64_t*)sc.get(sizeof(int64_t) * (mc + 1));
    cl.ne = (int64_t*)sc.get(sizeof(int64_t) * (mc + 1));
    cl.parent = (int64_t*)sc.get(sizeof(int64_t) * (mc + 1));
    cl.voff = (int64_t*)sc.get(sizeof(int64_t) * (mc + 2));
    cl.rep = (int32_t*)sc.get(sizeof(int32_t) * (mc + 1));
    int64_t* brings = lsup;  // free by now, [mc]
    int64_t* bat = psup;     // [mc + 1]
    int64_t* d_tot = (int64_t*)sc.get(sizeof(int64_t) * 2);
    if (!la.croot || !la.best || !la.ecount || !la.clid || !la.clstamp || !cl.c || !cl.nv || !cl.ne || !cl.parent ||
        !cl.voff || !cl.rep || !d_tot)
        return failed("hierarchy");
    RTR_CUDA_TRY(cudaMemsetAsync(la.best, 0xff, sizeof(int32_t) * (m + 1), rs));
    RTR_CUDA_TRY(cudaMemsetAsync(la.ecount, 0, sizeof(uint32_t) * (m + 1), rs));
    RTR_CUDA_TRY(cudaMemsetAsync(la.clstamp, 0xff, sizeof(int32_t) * (m + 1), rs));
    k_nuc_iota<<<gm, kBlock, 0, rs>>>(comp, m);
    g->launches += 3 + take_primitive_launches();
    RTR_CUDA_TRY(cudaStreamSynchronize(rs));
    std::vector<int64_t> first((size_t)max_c + 2, 0);  // c -> its first deletion
    for (int64_t c = 1; c <= max_c; ++c) first[c] = first[c - 1] + per_level[c - 1];
    int64_t ncl = 0, vn = 0, vcap = 2 * (n + mc) + 64;
    int32_t* vert = (int32_t*)sc.get(sizeof(int32_t) * (size_t)(vcap + 1));
    if (!vert) return failed("members");
    for (int64_t c = max_c; c >= 2; --c) {  // kappa = c - 1; kappa 0 has no clusters
        la.cnt = per_level[c];
        if (la.cnt == 0) continue;
        la.lv = (int32_t)(c - 1);
        la.ord = ord + first[c];
        const int gl = grid_for(la.cnt, kBlock), gk = grid_for(ncl, kBlock);
        k_nuc_join<<<gl, kBlock, 0, rs>>>(la);
        k_nuc_comps<<<gl, kBlock, 0, rs>>>(la);
        k_nuc_roots<<<gl, kBlock, 0, rs>>>(la);
        RTR_TRY(exclusive_scan_u32(la.is_start, hpos, la.cnt, next + 6, stmp, rs));
        k_nuc_clusters<<<gl, kBlock, 0, rs>>>(la, hpos, ncl, cl);
        RTR_CUDA_TRY(cudaMemsetAsync(d_tot, 0, sizeof(int64_t) * 2, rs));
        if (ncl > 0) {
            k_nuc_children<<<gk, kBlock, 0, rs>>>(la, ncl, cl, brings);
            g->launches += 1;
            RTR_TRY(exclusive_scan_i64(brings, bat, ncl, d_tot, ltmp, rs));
        }
        unsigned born = 0;
        int64_t brought = 0;
        RTR_CUDA_TRY(cudaMemcpyAsync(&born, next + 6, sizeof born, cudaMemcpyDeviceToHost, rs));
        RTR_CUDA_TRY(cudaMemcpyAsync(&brought, d_tot, sizeof brought, cudaMemcpyDeviceToHost, rs));
        RTR_CUDA_TRY(cudaStreamSynchronize(rs));
        const int64_t cnt = 2 * la.cnt + brought;
        if (cnt >= (1ll << 32)) {
            set_error("a nucleus level has %lld member entries", (long long)cnt);
            return RTR_ERR_LIMIT;
        }
        Scratch lsc(r);
        uint64_t* mk = (uint64_t*)lsc.get(sizeof(uint64_t) * (cnt + 1));
        uint64_t* ma = (uint64_t*)lsc.get(sizeof(uint64_t) * (cnt + 1));
        void* mt = lsc.get(radix_temp_bytes(cnt));
        uint32_t* mflag = (uint32_t*)lsc.get(sizeof(uint32_t) * (cnt + 1));
        uint32_t* mpos = (uint32_t*)lsc.get(sizeof(uint32_t) * (cnt + 1));
        uint32_t* mtmp = (uint32_t*)lsc.get(sizeof(uint32_t) * scan_temp_elems(cnt + 1));
        if (!mk || !ma || !mt || !mflag || !mpos || !mtmp) return failed("members");
        const int gq = grid_for(cnt, kBlock);
        k_nuc_edge_members<<<gl, kBlock, 0, rs>>>(la, ncl, B, mk);
        if (brought > 0) {
            k_nuc_child_members<<<grid_for(32 * ncl, kBlock), kBlock, 0, rs>>>(ncl, cl, brings, bat, vert, B,
                                                                               mk + 2 * la.cnt);
            g->launches += 1;
        }
        uint64_t* ms = nullptr;
        RTR_TRY(radix_sort_u64(mk, ma, cnt, B + bits_for((uint64_t)born), mt, rs, &ms));
        k_nuc_distinct<<<gq, kBlock, 0, rs>>>(ms, cnt, mflag);
        RTR_TRY(exclusive_scan_u32(mflag, mpos, cnt, next + 7, mtmp, rs));
        unsigned distinct = 0;
        RTR_CUDA_TRY(cudaMemcpyAsync(&distinct, next + 7, sizeof distinct, cudaMemcpyDeviceToHost, rs));
        RTR_CUDA_TRY(cudaStreamSynchronize(rs));
        if (vn + distinct > vcap) {  // more room for the members, kept
            const int64_t want = 2 * (vn + (int64_t)distinct) + 64;
            int32_t* more = (int32_t*)sc.get(sizeof(int32_t) * (size_t)(want + 1));
            if (!more) return failed("members");
            RTR_CUDA_TRY(cudaMemcpyAsync(more, vert, sizeof(int32_t) * (size_t)vn, cudaMemcpyDeviceToDevice, rs));
            vert = more;
            vcap = want;
        }
        k_nuc_members<<<gq, kBlock, 0, rs>>>(ms, cnt, mflag, mpos, next + 7, ncl, B, vn, cl, vert);
        k_nuc_sizes<<<grid_for(born, kBlock), kBlock, 0, rs>>>(ncl, ncl + born, cl);
        g->launches += 8 + take_primitive_launches();
        RTR_CUDA_TRY(cudaGetLastError());
        ncl += born;
        vn += distinct;
    }
    g->nuc_c.resize(ncl);
    g->nuc_nv.resize(ncl);
    g->nuc_ne.resize(ncl);
    g->nuc_parent.resize(ncl);
    g->nuc_off.resize(ncl + 1);
    g->nuc_vert.resize(vn);
    if (ncl > 0) {
        const size_t bytes = sizeof(int64_t) * (size_t)ncl;
        RTR_CUDA_TRY(cudaMemcpyAsync(g->nuc_c.data(), cl.c, bytes, cudaMemcpyDeviceToHost, rs));
        RTR_CUDA_TRY(cudaMemcpyAsync(g->nuc_nv.data(), cl.nv, bytes, cudaMemcpyDeviceToHost, rs));
        RTR_CUDA_TRY(cudaMemcpyAsync(g->nuc_ne.data(), cl.ne, bytes, cudaMemcpyDeviceToHost, rs));
        RTR_CUDA_TRY(cudaMemcpyAsync(g->nuc_parent.data(), cl.parent, bytes, cudaMemcpyDeviceToHost, rs));
        RTR_CUDA_TRY(cudaMemcpyAsync(g->nuc_off.data(), cl.voff, bytes, cudaMemcpyDeviceToHost, rs));
        int64_t* mv = (int64_t*)sc.get(sizeof(int64_t) * (size_t)(vn + 1));
        if (!mv) return failed("labels");
        k_nuc_labels<<<grid_for(vn, kBlock), kBlock, 0, rs>>>(vert, vn, inv, mv);
        g->launches += 1;
        RTR_CUDA_TRY(cudaGetLastError());
        RTR_CUDA_TRY(cudaMemcpyAsync(g->nuc_vert.data(), mv, sizeof(int64_t) * (size_t)vn, cudaMemcpyDeviceToHost, rs));
    }
    RTR_CUDA_TRY(cudaStreamSynchronize(rs));
    g->nuc_off[ncl] = vn;
    g->nuc_done = true;
    return RTR_OK;
}

}  // namespace

extern "C" {

int rtr_nucleus(rtr_graph* g, int64_t* n_clusters)
{
    if (!g) {
        set_error("null graph");
        return RTR_ERR_ARG;
    }
    if (g->stage < 1) {
        set_error("nucleus called before the graph was built");
        return RTR_ERR_STATE;
    }
    if (g->nbatch > 0) {
        set_error("the nucleus path is not defined for a batch handle");
        return RTR_ERR_ARG;
    }
    RTR_CUDA_TRY(cudaSetDevice(g->device));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, g->stream);
    const int rc = nucleus_run(g);
    cudaEventRecord(e1, g->stream);
    cudaEventSynchronize(e1);
    cudaEventElapsedTime(&g->ms_nucleus, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    if (n_clusters) *n_clusters = (int64_t)g->nuc_c.size();
    return RTR_OK;
}

int rtr_get_nuclei(const rtr_graph* g, int64_t* n_clusters, int64_t* n_members, int64_t* c, int64_t* nv,
                   int64_t* ne, int64_t* parent, int64_t* off, int64_t* vert)
{
    if (!g || !g->nuc_done) {
        set_error("the nucleus path has not run on this graph");
        return RTR_ERR_STATE;
    }
    const size_t k = g->nuc_c.size();
    if (n_clusters) *n_clusters = (int64_t)k;
    if (n_members) *n_members = (int64_t)g->nuc_vert.size();
    if (c) std::copy(g->nuc_c.begin(), g->nuc_c.end(), c);
    if (nv) std::copy(g->nuc_nv.begin(), g->nuc_nv.end(), nv);
    if (ne) std::copy(g->nuc_ne.begin(), g->nuc_ne.end(), ne);
    if (parent) std::copy(g->nuc_parent.begin(), g->nuc_parent.end(), parent);
    if (off) std::copy(g->nuc_off.begin(), g->nuc_off.end(), off);
    if (vert) std::copy(g->nuc_vert.begin(), g->nuc_vert.end(), vert);
    return RTR_OK;
}

int rtr_write_nuclei(const rtr_graph* g, const char* path)
{
    if (!g || !path || !g->nuc_done) {
        set_error("null argument, or the nucleus path has not run on this graph");
        return !g || !path ? RTR_ERR_ARG : RTR_ERR_STATE;
    }
    FILE* f = fopen(path, "w");
    if (!f) {
        set_error("could not open %s for writing", path);
        return RTR_ERR_IO;
    }
    std::string line;
    for (size_t k = 0; k < g->nuc_c.size(); ++k) {
        char head[160];
        snprintf(head, sizeof head, "Cluster id: %lld, C: %lld, n_vertices: %lld, n_edges: %lld, parent: %lld\n",
                 (long long)k, (long long)g->nuc_c[k], (long long)g->nuc_nv[k], (long long)g->nuc_ne[k],
                 (long long)g->nuc_parent[k]);
        line.assign(head);
        for (int64_t p = g->nuc_off[k]; p < g->nuc_off[k + 1]; ++p) {
            line += std::to_string(g->nuc_vert[p]);
            line += ' ';
        }
        line += '\n';
        if (fwrite(line.data(), 1, line.size(), f) != line.size()) {
            fclose(f);
            set_error("short write to %s", path);
            return RTR_ERR_IO;
        }
    }
    if (fclose(f) != 0) {
        set_error("could not close %s", path);
        return RTR_ERR_IO;
    }
    return RTR_OK;
}

}  // extern "C"
