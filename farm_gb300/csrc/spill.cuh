// Work sharing for the pair kernels (intersect, contain, within): pixel pairs
// that a warp leaves to all warps.
//
// A persistent warp per candidate pair is the cheapest way through a list of
// light pairs, but a pair of two heavy polygons has up to 10^6 times a light
// one's segment tests, and a list that is short, or uneven, then waits for a
// few warps. So a warp spends a bounded number of (estimated) segment tests on
// a pair and spills the pixel pairs that are left to a pool, from which a
// second kernel's warps take them one by one. 57,051 pairs of polygons of up
// to 100,000 vertices at -v 64: 158 ms with a warp per pair, 11 ms so.
#pragma once

#include "common.cuh"

namespace farm {

constexpr int kQueue = 256;             // pixel pairs buffered per warp, and per chunk of the pool
constexpr float kShareTests = 16384.f;  // estimated segment tests above which a spilled pixel pair is shared

// A chunk of the pool: up to kQueue pixel pairs of one candidate pair.
struct SpillChunk {
    uint64_t pid;
    uint32_t head;   // the pair's first chunk: its flag says the pair is decided
    uint32_t count;  // pixel pairs
    uint32_t parts;  // shares each is cut into
    uint32_t pad;
};
struct SpillPool {
    uint2 *items = nullptr;  // kQueue per chunk
    SpillChunk *chunk = nullptr;
    uint32_t *flag = nullptr;  // per chunk (heads only): the pair is decided
    unsigned long long *ctr = nullptr;  // [0] chunks asked for, [1] next unit, [2] most units of a chunk; zeroed
    uint32_t cap = 0;   // chunks in the pool; 0: every pair stays with its warp
    float budget = 0;   // estimated segment tests a warp spends on a pair before it spills the rest
};

// Segment tests of an average pixel pair: edges and sequences per pixel of both sides.
__device__ __forceinline__ float pixel_pair_cost(const PolyHdr &S, const PolyHdr &T) {
    return ((float)S.nv + (float)S.n_seq) / (float)S.P * (((float)T.nv + (float)T.n_seq) / (float)T.P);
}

// The warp's queue entries [k, n) into a chunk of the pool; false when it is
// full. *head / *spilled are the pair's (warp-uniform).
__device__ __forceinline__ bool spill_rest(const SpillPool &sp, uint64_t pid, const uint2 *q, int k, int n,
                                           float cost, int lane, uint32_t *head, bool *spilled) {
    unsigned long long c = 0;
    if (lane == 0) c = atomicAdd(&sp.ctr[0], 1ull);
    c = __shfl_sync(0xffffffffu, c, 0);
    if (c >= sp.cap) return false;
    for (int e = k + lane; e < n; e += 32) sp.items[c * kQueue + (e - k)] = q[e];
    if (!*spilled) *head = (uint32_t)c;
    *spilled = true;
    if (lane == 0) {
        const float share = cost / kShareTests;
        const uint32_t parts = share <= 1.f ? 1u : (share >= 16.f ? 16u : (uint32_t)share);
        sp.chunk[c] = SpillChunk{pid, *head, (uint32_t)(n - k), parts, 0u};
        sp.flag[c] = 0u;
        atomicMax(&sp.ctr[2], (unsigned long long)(n - k) * parts);
    }
    return true;
}

// Take the pool's pixel pairs over all warps of the grid: f(pid, entry, part,
// parts) returns true (warp-uniform) when it decides the pair, done(pid) runs
// once, on lane 0, for a pair that was decided. A unit is a share of one
// entry; units are taken entry by entry across the chunks (unit u belongs to
// chunk u % n), so that with many spilled pairs each pair's first entries
// still come first and a decided pair stops early, and with few of them every
// warp works on the same pair.
template <typename F, typename D>
__device__ __forceinline__ void spill_units(const SpillPool &sp, F f, D done) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned long long n = min(sp.ctr[0], (unsigned long long)sp.cap);
    if (n == 0) return;
    const unsigned long long total = n * sp.ctr[2];
    // units per grab: one while units are scarce, up to a warp's worth
    const unsigned long long warps = (unsigned long long)gridDim.x * (blockDim.x >> 5);
    const unsigned long long grab = min(32ull, max(1ull, total / (16ull * warps)));
    for (;;) {
        unsigned long long u = 0;
        if (lane == 0) u = atomicAdd(&sp.ctr[1], grab);
        u = __shfl_sync(full, u, 0);
        if (u >= total) break;
        u += lane;
        uint32_t c = 0, v = 0, head = 0, parts = 1;
        unsigned long long pid = 0;
        bool valid = (unsigned long long)lane < grab && u < total;
        if (valid) {
            c = (uint32_t)(u % n);
            v = (uint32_t)(u / n);
            const SpillChunk h = sp.chunk[c];
            head = h.head;
            parts = h.parts;
            pid = h.pid;
            valid = v < h.count * h.parts;
        }
        for (unsigned m = __ballot_sync(full, valid); m; m &= m - 1) {
            const int src = __ffs(m) - 1;
            const uint32_t hd = __shfl_sync(full, head, src);
            if (__shfl_sync(full, *(volatile uint32_t *)&sp.flag[hd], 0)) continue;  // the pair is decided
            const unsigned long long p = __shfl_sync(full, pid, src);
            const uint32_t np = __shfl_sync(full, parts, src), vv = __shfl_sync(full, v, src);
            const uint2 e = sp.items[(uint64_t)__shfl_sync(full, c, src) * kQueue + vv / np];
            if (f(p, e, vv % np, np) && lane == 0 && atomicExch(&sp.flag[hd], 1u) == 0u) done(p);
        }
    }
}

// A pool for a call over n pairs in the store's scratch, its counters at
// ctr[0..2] (zeroed by the caller): 4,096 to 65,536 chunks of 2 KB, when it is
// full, warps keep what is left of their pairs. The budget is `few` up to a
// pair per resident warp, where the longest pair is the whole wait, and `many`
// beyond. FARM_SPILL_BUDGET sets it.
int spill_pool(farm_store *s, uint64_t n, unsigned long long *ctr, float few, float many, SpillPool *sp);

// Work order of a pair list: by descending product of the polygons' vertex
// counts, so that the heaviest pairs start first and the pass does not end on a
// long pair that started last. Results are written by pair index, so the order
// is invisible. *order is null (index order) for a list of up to a pair per
// resident warp, whose pairs all start at once. FARM_PAIR_ORDER=0: index order.
int pair_order(farm_store *s, const uint32_t *dpairs, uint64_t n, uint64_t tgt_base, const uint32_t **order);

}  // namespace farm
