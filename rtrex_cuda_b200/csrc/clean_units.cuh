// Types shared by the two replays of the cascading clean: the warp-per-unit
// replay (clean.cu) and the round-parallel replay of large units
// (clean_rounds.cu).
#pragma once

#include "rtr_graph.cuh"

namespace rtr {

// One unit of the clean: a connected component of the triangle-carrying
// edges, with its seeds (sorted seed range) and its cascade-stack region.
struct UnitDesc {
    int64_t seed_begin;
    int64_t seed_end;
    int64_t stack_base;
    int64_t stack_cap;
    int64_t root;  // the unit's union-find root (smallest vertex id)
    int64_t edges;  // its triangle-carrying edges
};

// One cascade-stack entry: the pair as deleteAndClean pushed it plus the
// static data its pop needs (degrees, triangle-list bounds), so a pop issues
// no lookups before its first dynamic load.  Seeds use the same descriptor.
struct StackEntry {
    int32_t e;        // forward rank of the edge
    int32_t first;    // Pair.first  (deleteAndClean's u)
    int32_t second;   // Pair.second (deleteAndClean's v)
    int32_t dfirst;   // deg(first)
    int32_t dsecond;  // deg(second)
    int32_t cnt;      // triangle-list length
    int64_t t0;       // triangle-list start
};
static_assert(sizeof(StackEntry) == 32, "StackEntry is 32 bytes");

// Streaming read of a triangle-list entry: the clean reads each list once, so
// entries are loaded evict-first and do not displace the edge records in L2.
__device__ __forceinline__ TriEntry ld_entry(const TriEntry* p)
{
    TriEntry t;
    int4* d = reinterpret_cast<int4*>(&t);
    d[0] = __ldcs(reinterpret_cast<const int4*>(p));
    d[1] = __ldcs(reinterpret_cast<const int4*>(p) + 1);
    return t;
}

// Orientation of a popped pair (u, v) as deleteAndClean sees it
// (Decomposition.h:178-186): the lower-degree endpoint's list is scanned.
struct PairSide {
    bool lower_is_a;  // lower == the smaller vertex id (the forward edge's a)
    int32_t lower, higher, dlow, dhigh;
};

__device__ __forceinline__ PairSide pair_side(const StackEntry& c)
{
    const bool lo_is_u = c.dfirst < c.dsecond;
    PairSide s;
    s.lower = lo_is_u ? c.first : c.second;
    s.higher = lo_is_u ? c.second : c.first;
    s.dlow = lo_is_u ? c.dfirst : c.dsecond;
    s.dhigh = lo_is_u ? c.dsecond : c.dfirst;
    s.lower_is_a = s.lower == (c.first < c.second ? c.first : c.second);
    return s;
}

// One pop of the window replay.
struct alignas(16) PopLog {
    int32_t e;   // forward rank of its edge (-1: unused)
    int32_t n;   // live triangles it removed
    int64_t at;  // its triangle list
};

// How a unit is replayed, in the schedule's order: in windows of long or of short
// triangle lists, each for units of many seeds and of few, or by one warp.
enum UnitClass : uint32_t { UNIT_WIDE = 0, UNIT_WIDE_FEW, UNIT_NARROW, UNIT_NARROW_FEW, UNIT_WARP, UNIT_KINDS };

// Window replay (clean_rounds.cu) of the units at the front of `order`, kinds[k] of
// each kind in turn: one thread block per unit on the kind's stream,
// concurrently with whatever the caller launches on the graph's stream; the
// popped edges' perEdge and the per-vertex weights of those units are folded in
// afterwards, in the reference's order, by clean_rounds_finish on the graph's
// stream (after the others are joined).
struct RoundReplay {
    EdgeRec* rec = nullptr;
    int64_t pops_cap = 0, logs_cap = 0;
    PopLog* plog = nullptr;
    uint8_t* live8 = nullptr;  // per list entry: its triangle was removed by the pop of its list's edge
    // the fold's: per pop, per removed triangle, per subtraction
    uint32_t *pcnt = nullptr, *poff = nullptr, *ptmp = nullptr;
    double* wlog = nullptr;
    uint64_t *keys = nullptr, *alt = nullptr;
    void* rtmp = nullptr;
    double* ws = nullptr;
    longlong2* runs = nullptr;
    unsigned* nruns = nullptr;
};
// The memory of all that, before anything is replayed: about 85 bytes for each
// triangle of the units, beside the lists' 96.  False when it does not fit: the
// units then replay one warp each, which needs none of it (the lists are kept
// without regard to the log, so no graph loses its clean to it).
bool clean_rounds_reserve(rtr_graph* g, Scratch& sc, int64_t stack_entries, int64_t log_entries, RoundReplay* rr);
int clean_rounds_launch(rtr_graph* g, const cudaStream_t* st, EdgeRec* rec, const StackEntry* seeds,
                        const UnitDesc* units, const uint64_t* order, const int64_t* kinds, StackEntry* stacks,
                        RoundReplay* rr);
int clean_rounds_finish(rtr_graph* g, RoundReplay* rr);

}  // namespace rtr
