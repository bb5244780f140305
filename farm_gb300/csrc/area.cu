// Stage (d): FP64 intersection area of candidate pairs.
//
// The reference stops before computing any area (Ideal.cpp:1683; its GPU
// rebuild step is never launched, query_intersection.cu:724-737), so this is
// the project's own formulation, checked against the FP64 CPU oracle.
//
// Boundary integral: area(A n B) = 1/2 * [ integral over the parts of dA inside
// B + over the parts of dB inside A ] of (x dy - y dx), each boundary taken
// with its own orientation sign. Along a straight edge P -> Q (d = Q - P) the
// integrand is the constant P x d per unit of the edge parameter, so an edge
// contributes (P x d) * (total parameter length of its inside parts). Those
// parts are delimited by the edge's crossings with the other boundary; the
// state at a chunk's first vertex comes from one point-in-polygon test on the
// other polygon's raster, and flips at each crossing after it.
//
// Work: items are (pair, side, chunk of that side's edges), taken by persistent
// warps from a global counter. A lane holds one edge; the warp walks the window
// of the other polygon's raster around all its edges together and queues the
// edges listed there whose box meets the group's (each at its first listing);
// the lanes test their edges against the queued ones, a group of fewer than 32
// edges in slices that share the queue. An edge's share is its signed inside
// length: the leaving parameters minus the entering ones, plus the tail when it
// ends inside. Per-item partial sums are reduced per pair in a fixed order
// (deterministic results).
// Coordinates are taken relative to the pair's source first vertex.
// General position is assumed (no collinear overlaps, no crossing exactly at a
// vertex); crossings at a shared vertex are counted once by half-open ranges.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"
#include "segments.cuh"

namespace farm {

// The tuning knob of the area pass by size bucket (bucket b holds pairs whose
// larger edge count has floor(log2) == b), chosen by farm_area_autotune: the
// edges per work item (default 32).
struct Chunks {
    uint16_t c[32];
    __host__ __device__ static int bucket(uint32_t es, uint32_t et) {
        uint32_t m = es > et ? es : et;
        return m ? 31 - clz32(m) : 0;
    }
    __host__ __device__ uint32_t of(uint32_t es, uint32_t et) const { return c[bucket(es, et)]; }
    __host__ __device__ static int clz32(uint32_t x) {
#ifdef __CUDA_ARCH__
        return __clz(x);
#else
        return __builtin_clz(x);
#endif
    }
};

// Items whose window holds many listings are cut into parts for all warps (see
// k_area). A chunk of the pool is such an item's state: the sums of its edges'
// crossings so far, the side of its first vertex, and its parts.
struct AreaSpill {
    unsigned long long sum[32];
    uint32_t cnt[32];
    uint64_t item;
    uint32_t state, parts, done;
    uint32_t pad;
};
struct AreaPool {
    AreaSpill *chunk = nullptr;
    uint2 *unit = nullptr;              // chunk, part; kAreaParts per chunk
    unsigned long long *ctr = nullptr;  // [0] chunks asked for, [1] units, [2] next unit; zeroed
    uint32_t cap = 0;                   // chunks; 0: every item stays with its warp
};
constexpr uint32_t kAreaParts = 32;   // most parts of an item
// Steps (32 sequences each) a warp takes of an item before it is cut, and of
// its parts. 801 pairs of up to 20,000 vertices: 5.16 ms; 32 / 8 5.38, 128 / 8
// 5.02, 64 / 4 5.36, 64 / 16 5.25 (6.7 to 9.8 where the pool is too small for
// the items cut); 1,440 pairs of up to 1,024 vertices: 1.35 ms with each.
constexpr uint32_t kAreaBudget = 64, kAreaShareSteps = 8;

struct AreaArgs {
    const uint32_t *pairs;
    const uint64_t *n;           // pair count (device scalar)
    uint64_t tgt_base;
    Chunks chunks;               // edges per item, by size bucket
    const uint64_t *item_start;  // per pair: first item; item_start[*n] = item count
    uint64_t cap_items;          // partial's capacity
    double *partial;             // per item
    const int8_t *orient;        // per polygon: +1 counter-clockwise, -1 clockwise
    const uint64_t *ep_off;      // per ring position: first entry of the edge's pixel list
    const uint32_t *ep_pix;      // pixels listing each edge (edge -> pixel CSR)
    unsigned long long *next;
    unsigned long long *overflow;  // [0] unused, [1] items beyond cap_items
    unsigned long long *work;      // [0] FP64 crossing tests, [1] crossings counted
    int spread;                    // take items in a spread order (see k_area)
    AreaPool pool;
    int rest;                      // the pool's parts instead of the items
};

// Crossing parameters are added as integers of 2^-60: exact, in any order and
// over any lanes. Entering and leaving ones alternate along an edge where the
// other ring is simple, so their signed sum lies in [-1, 1]; what partial sums
// carry beyond 64 bits falls off.
constexpr double kParamScale = 1152921504606846976.0;  // 2^60

__device__ __forceinline__ double cross2(double ax, double ay, double bx, double by) { return ax * by - ay * bx; }

// The other polygon's box and pixel size, in FP32: the box's corner in two
// parts, so that a difference from it is as good as one taken in FP64 and
// rounded, and its sides rounded so that a float is outside of them exactly
// when it is outside of the box.
struct Frame {
    float xh, xl, yh, yl, sx, sy;
    float x0, y0, x1, y1;
};
__device__ __forceinline__ Frame frame_of(const PolyHdr &O) {
    Frame f;
    f.xh = (float)O.mbr[0];
    f.xl = (float)(O.mbr[0] - f.xh);
    f.yh = (float)O.mbr[1];
    f.yl = (float)(O.mbr[1] - f.yh);
    f.sx = (float)O.step_x;
    f.sy = (float)O.step_y;
    f.x0 = __double2float_ru(O.mbr[0]);
    f.y0 = __double2float_ru(O.mbr[1]);
    f.x1 = __double2float_rd(O.mbr[2]);
    f.y1 = __double2float_rd(O.mbr[3]);
    return f;
}

// Point-in-polygon of a vertex for polygon H through its raster, by a warp: a
// ray to the right along the pixel row; the first non-BORDER pixel tells its
// side, edges of BORDER pixels before it flip the parity (each edge counted in
// the pixel whose x-range holds its crossing). The pixel and the crossing are
// decided in FP32 when the pixel's ends and the point are further off than the
// rounding (10 u of the box's coordinates at most), else in FP64.
__device__ bool pip_raster(const StoreView &sv, const PolyHdr &H, const Frame &fr, float2 pt, int cc, int lane) {
    if (pt.x < fr.x0 || pt.x > fr.x1 || pt.y < fr.y0 || pt.y > fr.y1) return false;
    const float u = ((pt.x - fr.xh) - fr.xl) / fr.sx, v = ((pt.y - fr.yh) - fr.yl) / fr.sy;
    int col = (int)u, row = (int)v;
    const float fu = u - (float)col, fv = v - (float)row, mu = 1e-4f + 1e-6f * u, mv = 1e-4f + 1e-6f * v;
    if (!(fu > mu && fu < 1.f - mu && col < H.dimx)) col = offset_x(H.mbr, H.step_x, H.dimx, pt.x);
    if (!(fv > mv && fv < 1.f - mv && row < H.dimy)) row = offset_y(H.mbr, H.step_y, H.dimy, pt.y);
    const uint8_t *st = sv.status + H.st;
    const uint32_t *off = sv.offset + H.off;
    const uint2 *seq = sv.seq + H.seq;
    const float2 *r = sv.ring + H.ring;
    const float m = 1e-6f * (fabsf(fr.x0) + fabsf(fr.x1)) + 1.2e-38f;
    bool odd = false;
#pragma unroll 1
    for (int c = col; c < H.dimx; c++) {
        const uint32_t pid = (uint32_t)(row * H.dimx + c);
        const int s = show_status(st[pid], cc);
        if (s != 1) return c == col ? (s == 2) : (odd ^ (s == 2));
        const float lo = c == col ? pt.x : fmaxf(pt.x, fr.xh + (float)c * fr.sx);
        const float hi = c == H.dimx - 1 ? INFINITY : fr.xh + (float)(c + 1) * fr.sx;
        bool flip = false;
#pragma unroll 1
        for (uint32_t q = off[pid] + lane; q < off[pid + 1]; q += 32) {
            const uint2 sq = seq[q];
#pragma unroll 1
            for (uint32_t k = 0; k < sq.y; k++) {
                const float2 a = r[sq.x + k], b = r[sq.x + k + 1];
                if ((a.y > pt.y) == (b.y > pt.y)) continue;
                const float dx = b.x - a.x, dy = b.y - a.y;
                const float xf = a.x + (pt.y - a.y) / dy * dx;
                const bool ok = fabsf(dy) < INFINITY;
                if (ok && (xf < lo - m || xf > hi + m)) continue;
                bool in = ok && xf > lo + m && xf < hi - m;
                if (!in) {
                    const double x_lo = c == col ? -1e300 : H.mbr[0] + c * H.step_x;
                    const double x_hi = c == H.dimx - 1 ? 1e300 : H.mbr[0] + (c + 1) * H.step_x;
                    const double xi = (double)a.x + ((double)pt.y - a.y) * ((double)b.x - a.x) / ((double)b.y - a.y);
                    in = xi > (double)pt.x && xi >= x_lo && xi < x_hi;
                }
                if (in) flip = !flip;
            }
        }
        odd ^= __popc(__ballot_sync(0xffffffffu, flip)) & 1;
    }
    return odd;  // past the raster: outside, so the crossings decide
}

// An edge in the other polygon's pixel units, with the rounding of those: m is
// far above it.
struct EdgeUV {
    float u0, v0, u1, v1, m;
    float per_row;  // 1 / (v1 - v0), 0 when that is within m
};
__device__ __forceinline__ EdgeUV edge_uv(const Frame &O, float2 P, float2 Q) {
    EdgeUV e;
    e.u0 = ((P.x - O.xh) - O.xl) / O.sx;
    e.v0 = ((P.y - O.yh) - O.yl) / O.sy;
    e.u1 = ((Q.x - O.xh) - O.xl) / O.sx;
    e.v1 = ((Q.y - O.yh) - O.yl) / O.sy;
    e.m = 0.01f + 1e-6f * fmaxf(fmaxf(fabsf(e.u0), fabsf(e.u1)), fmaxf(fabsf(e.v0), fabsf(e.v1)));
    e.per_row = fabsf(e.v1 - e.v0) > e.m ? 1.f / (e.v1 - e.v0) : 0.f;
    return e;
}

// Columns of row y searched for edges that may cross edge e: those the edge
// spans within rows y - 1 .. y + 1 and one more on either side, every pixel
// within a pixel of its path. That holds every edge of O that it crosses (an
// edge is listed in each pixel it passes through, or, where the reference's
// walk cuts a grid corner, in the diagonal neighbours). lo > hi: none.
__device__ __forceinline__ int2 edge_columns(const EdgeUV &e, int y, int dimx) {
    const float a = (float)(y - 1) - e.m, b = (float)(y + 2) + e.m;
    if (fmaxf(e.v0, e.v1) < a || fminf(e.v0, e.v1) > b) return make_int2(0x7fffffff, -1);
    const float du = e.u1 - e.u0;
    float t0 = 0.f, t1 = 1.f;
    if (e.per_row != 0.f) {
        const float p = (a - e.v0) * e.per_row, q = (b - e.v0) * e.per_row;
        t0 = fmaxf(0.f, fminf(p, q));
        t1 = fminf(1.f, fmaxf(p, q));
    }
    const float p = e.u0 + t0 * du, q = e.u0 + t1 * du;
    const float lo = floorf(fminf(p, q) - e.m) - 1.f, hi = floorf(fmaxf(p, q) + e.m) + 1.f;
    const int l = lo > 0.f ? (lo < 2e9f ? (int)lo : 0x7fffffff) : 0;
    const int h = hi < (float)(dimx - 1) ? (hi >= 0.f ? (int)hi : -1) : dimx - 1;
    return l <= h ? make_int2(l, h) : make_int2(0x7fffffff, -1);
}

// whether the edge has a length and its box meets O's
__device__ __forceinline__ bool edge_meets(const Frame &O, float2 P, float2 Q) {
    return (P.x != Q.x || P.y != Q.y) && !(fmaxf(P.x, Q.x) < O.x0 || fminf(P.x, Q.x) > O.x1 ||
                                           fmaxf(P.y, Q.y) < O.y0 || fminf(P.y, Q.y) > O.y1);
}

// A group of up to 32 consecutive edges [first, first + n) of a ring, searched
// together: the window's columns of row y are those between the first and the
// last that any of them searches.
struct Group {
    const PolyHdr *O;
    const float2 *ring;
    uint32_t first, n;
    int sy;
};
constexpr int kRowCache = 256;  // a window's last rows, kept by row & (kRowCache - 1)
constexpr int kQueueRows = 64;  // rows a queued edge may wait
// the group's columns of a row that is no longer kept
__device__ __noinline__ int2 group_columns(const Group &g, int y) {
    int2 c = make_int2(0x7fffffff, -1);
    const Frame fr = frame_of(*g.O);
#pragma unroll 1
    for (uint32_t k = 0; k < g.n; k++) {
        const float2 P = g.ring[g.first + k], Q = g.ring[g.first + k + 1];
        if (!edge_meets(fr, P, Q)) continue;
        const int2 e = edge_columns(edge_uv(fr, P, Q), y, g.O->dimx);
        c.x = min(c.x, e.x);
        c.y = max(c.y, e.y);
    }
    return c;
}

// Whether the listing of edge f in pixel pid (sequence q; lo: its row's first
// column) is the first listing of f in the group's window: no BORDER pixel of
// the window with a smaller id (an earlier row, or the same row further left)
// lists f, and no earlier sequence of pid holds it. Each edge that crosses is
// then counted exactly once, whatever the number of pixels listing it, with no
// per-edge memory. The pixels listing f come from the edge -> pixel index
// (ascending ids, so the scan stops at pid), window membership from the kept
// rows (or the same function for older ones).
__device__ bool first_listing(const StoreView &sv, const Group &g, const int2 *rows, const uint64_t *ep_off,
                              const uint32_t *ep_pix, int cc, uint32_t pid, int lo, uint32_t q, uint32_t f) {
    const PolyHdr &O = *g.O;
    const uint64_t at = O.ring + f;
    const uint32_t dimx = (uint32_t)O.dimx;
    const int py = (int)(pid / dimx);
    int self = 0;
#pragma unroll 1
    for (uint64_t i = ep_off[at], e = ep_off[at + 1]; i < e; i++) {
        const uint32_t r = ep_pix[i];
        if (r > pid) break;
        if (r == pid) {
            self++;
            continue;
        }
        const int ry = (int)(r / dimx), rx = (int)(r - (uint32_t)ry * dimx);
        if (ry < g.sy) continue;  // above the window
        int2 c = make_int2(lo, 0x7fffffff);
        if (ry != py) c = ry > py - (kRowCache - kQueueRows) ? rows[ry & (kRowCache - 1)] : group_columns(g, ry);
        if (rx >= c.x && rx <= c.y && show_status(sv.status[O.st + r], cc) == 1) return false;
    }
    if (self > 1) {  // pid holds f in more than one sequence: the first counts
        const uint2 *seq = sv.seq + O.seq;
#pragma unroll 1
        for (uint32_t p = sv.offset[O.off + pid]; p < q; p++) {
            const uint2 sq = seq[p];
            if (f >= sq.x && f - sq.x < sq.y) return false;
        }
    }
    return true;
}

// Crossing parameter t of segment P -> Q with edge e of ring r, in [0, 1) on
// both (half-open, so a crossing at a shared vertex counts once); known: that
// they cross is certain, only t is wanted. The differences of floats are taken
// in double; both parameters' ranges are decided on numerator and denominator
// (n / d < 1 exactly when |n| < |d| of the same sign, as doubles one ulp apart
// divide to less than 1), so that only a crossing divides, once.
__device__ __forceinline__ bool crossing(float2 P, float2 Q, const float2 *r, uint32_t e, bool known, double &t,
                                         double &den) {
    const float2 a = r[e], b = r[e + 1];
    const double dx = (double)Q.x - P.x, dy = (double)Q.y - P.y;
    const double gx = (double)b.x - a.x, gy = (double)b.y - a.y;
    den = cross2(dx, dy, gx, gy);
    const double rx = (double)a.x - P.x, ry = (double)a.y - P.y;
    const double tn = cross2(rx, ry, gx, gy);
    if (!known) {
        if (den == 0) return false;
        const double un = cross2(rx, ry, dx, dy), ad = fabs(den);
        const bool neg = den < 0;
        const bool t_in = fabs(tn) < ad && (tn == 0 || (tn < 0) == neg);
        const bool u_in = fabs(un) < ad && (un == 0 || (un < 0) == neg);
        if (!(t_in && u_in)) return false;
    }
    t = tn / den;
    return true;
}

// Edges per item: one group, a lane each. 801 pairs of up to 20,000 vertices: 7.7
// ms with 8, 5.2 with 16, 4.5 with 24, 4.0 with 32; 1,440 pairs of up to 1,024
// vertices 1.55 / 1.38 / 1.41 / 1.37 ms. Larger items repeat no walk either, but
// are not cut.
constexpr int kDefaultChunk = 32;
constexpr int kDefaultWide = 200;   // of the window table, which nothing reads any more

// FARM_AREA_SPREAD=0 takes the items in pair order
static int spread_items() {
    const char *v = getenv("FARM_AREA_SPREAD");
    return (v && *v == '0') ? 0 : 1;
}


// What bounds it is instruction issue and the latency of the look-ups, then
// FP64, which GB300 issues at 1/64 of its FP32 rate. A lane per edge that
// walked its own window of pixels, sequences and listed edges kept 7 of 32
// lanes busy and took two FP64 divisions per row and edge; consecutive edges
// lie together, so the group's common window is little larger than each
// edge's, and its listings go through three queues, each worked off 32 at a
// time by all lanes: listings whose edge's box meets the group's (are they the
// edge's first?), the edges of first listings (FP32 test with every lane's
// edge), and the pairs that may cross (FP64). A group of R < 32 edges is
// repeated over floor(32 / R) slices of lanes in the test. Row ranges are FP32
// with a margin: they need only hold every crossing's listings, and the same
// for all of an item. A pair of edges is rejected in FP32 when one lies
// strictly on one side of the other's line by a margin far above the test's
// rounding and crossing()'s, and known to cross when both lie on either side
// by it.
//
// Items differ by three orders of magnitude: half of them take under 10 us,
// while an edge of a small polygon can have most of a large one in its window
// (20,000 listings, 5 ms, twice the whole pass's share of a warp). So an item
// is cut after kAreaBudget steps; a second launch takes the parts, each every
// parts-th step of the same walk, adds its integer sums to the item's, and the
// last one finishes the item: the same bits however it is cut.
// 801 pairs of up to 20,000 vertices: 72 ms with a window per lane, 10.0 ms
// with the look-up after the tests, 6.2 ms without cutting, 4.3 ms so, 3.7 ms
// with groups of 32 edges. Loops are not unrolled: most run once or twice, and
// the code is larger than the instruction cache takes lightly (77 KB unrolled,
// 70 KB so: 3.87 -> 3.68 ms). What a warp of the first launch waits for then is
// the look-ups' loads, with FP64 busy 44% of the time.
constexpr int kAreaQueue = 64;
struct AreaListing {  // an edge met in a pixel of the window
    uint32_t f, pid, q;
    int lo;  // first column of the row it was met in
};
// the warp's share of an item
struct AreaShare {
    AreaSpill *sp;         // the item's chunk, if it is in the pool
    uint32_t own, stride;  // its steps: own, own + stride, ...
    uint32_t left;         // some of the item is left to others
};

// The rest of the warp's item to the pool: false when that is full.
__device__ __noinline__ bool area_spill(const AreaPool &pool, AreaShare *sh, uint64_t item, bool state, float rest,
                                        int lane) {
    unsigned long long c = 0, u = 0;
    if (lane == 0) c = atomicAdd(&pool.ctr[0], 1ull);
    c = __shfl_sync(0xffffffffu, c, 0);
    if (c >= pool.cap) return false;
    AreaSpill *sp = &pool.chunk[c];
    const uint32_t parts = 1u + min(kAreaParts - 1u, (uint32_t)(rest / (float)kAreaShareSteps));
    if (lane == 0) {
        sp->item = item;
        sp->state = state;
        sp->parts = parts;
        sp->done = 0;
        u = atomicAdd(&pool.ctr[1], (unsigned long long)parts);
        sh->sp = sp;
        sh->left = 1;
    }
    u = __shfl_sync(0xffffffffu, u, 0);
    if (lane < (int)parts) pool.unit[u + lane] = make_uint2((uint32_t)c, (uint32_t)lane);
    __syncwarp();
    return true;
}

__global__ void __launch_bounds__(256, 3) k_area(const StoreView sv, AreaArgs a) {
    __shared__ int2 s_rows[8][kRowCache];
    __shared__ AreaListing s_list[8][kAreaQueue];
    __shared__ float4 s_seg[8][kAreaQueue];
    __shared__ uint32_t s_edge[8][kAreaQueue];
    __shared__ uint32_t s_hit[8][kAreaQueue];
    __shared__ uint8_t s_hedge[8][kAreaQueue];
    __shared__ uint32_t s_lo[8][32], s_hi[8][32];
    __shared__ uint32_t s_cnt[8][32];
    __shared__ AreaShare s_share[8];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int cc = sv.category_count;
    int2 *rows = s_rows[wib];
    AreaListing *list = s_list[wib];  // listings, until there are 32 to look up
    float4 *seg = s_seg[wib];         // the edges of first listings (ends, number), until there are 32 for the FP32 test
    uint32_t *edge = s_edge[wib];
    uint32_t *hit = s_hit[wib];       // pairs that may cross, until there are 32 for the FP64 test
    uint8_t *hedge = s_hedge[wib];
    unsigned long long my_tests = 0, my_cross = 0;
    for (;;) {
        const uint64_t n = *a.n;
        const uint64_t nitems = a.item_start[n];
        if (nitems > a.cap_items) {  // a plan's capacity was exceeded: report, compute nothing
            if (lane == 0 && blockIdx.x == 0 && threadIdx.x == 0) atomicExch(&a.overflow[1], 1ull);
            break;
        }
        unsigned long long it = 0;
        if (lane == 0) it = atomicAdd(a.rest ? &a.pool.ctr[2] : a.next, 1ull);
        it = __shfl_sync(full, it, 0);
        AreaShare *share = &s_share[wib];
        if (a.rest) {
            if (it >= a.pool.ctr[1]) break;
            const uint2 u = a.pool.unit[it];
            AreaSpill *sp = &a.pool.chunk[u.x];
            it = sp->item;
            if (lane == 0) *share = AreaShare{sp, kAreaBudget + u.y, sp->parts, 0u};
        } else if (lane == 0) {
            *share = AreaShare{nullptr, 0u, 1u, 0u};
        }
        __syncwarp();
        if (it >= nitems) break;
        // Items lie pair after pair, and the heavy pairs' items are each slow:
        // taken in that order, a heavy pair near the end leaves a tail. The
        // k-th item taken is item k * P mod nitems (P prime, coprime to
        // nitems: a bijection), which spreads every pair's items over the
        // pass. Each item writes its own partial, and the per-pair reduction
        // runs in item order, so the results do not depend on this order.
        if (a.spread && !a.rest) {
            const uint64_t P = (nitems % 1000003ull) ? 1000003ull : 999983ull;
            it = (unsigned long long)((it * P) % nitems);
        }
        uint32_t p = find_segment(a.item_start, (uint32_t)n, it);
        uint64_t rel = it - a.item_start[p];
        const PolyHdr &S = sv.hdr[a.pairs[2 * p]];
        const PolyHdr &T = sv.hdr[a.tgt_base + a.pairs[2 * p + 1]];
        uint32_t es = S.nv - 1, et = T.nv - 1;  // edges (the ring's last edge is the zero-length closing one)
        const uint32_t chunk = a.chunks.of(es, et);
        uint64_t cs = (es + chunk - 1) / chunk;
        bool side_t = rel >= cs;
        const PolyHdr &M = side_t ? T : S;  // the boundary integrated
        const PolyHdr &O = side_t ? S : T;  // the polygon it is clipped by
        uint32_t first = (uint32_t)((side_t ? rel - cs : rel) * chunk);
        uint32_t me = side_t ? et : es;
        uint32_t last = first + chunk < me ? first + chunk : me;
        const float2 *mr = sv.ring + M.ring, *orr = sv.ring + O.ring;
        const float2 o0 = sv.ring[S.ring];
        const double ox = o0.x, oy = o0.y;
        const double sign = a.orient[side_t ? a.tgt_base + a.pairs[2 * p + 1] : a.pairs[2 * p]];
        const Frame frame = frame_of(O);
        // state at the chunk's first vertex
        bool state = a.rest ? share->sp->state != 0 : pip_raster(sv, O, frame, mr[first], cc, lane);
        // only a single group's sums can be left to the pool
        const uint32_t limit = !a.rest && a.pool.cap && last - first <= 32 ? kAreaBudget : 0xffffffffu;
        double acc = 0;
        // a crossing leaves O when O's edge turns the way O's interior lies:
        // entering iff (d x g) has the opposite sign of O's orientation
        const bool inner_left = a.orient[side_t ? a.pairs[2 * p] : a.tgt_base + a.pairs[2 * p + 1]] > 0;
        const uint8_t *ost = sv.status + O.st;
        const uint32_t *ooff = sv.offset + O.off;
        const uint2 *oseq = sv.seq + O.seq;
#pragma unroll 1
        for (uint32_t b0 = first; b0 < last; b0 += 32) {
            const uint32_t R = min(32u, last - b0), G = 32u / R, slice = (uint32_t)lane / R;
            const uint32_t e = b0 + (uint32_t)lane % R;
            const float2 P = mr[e], Q = mr[e + 1];
            const bool active = slice < G && edge_meets(frame, P, Q);
            // per edge: leaving t minus entering t, crossings
            s_lo[wib][lane] = s_hi[wib][lane] = 0u;
            s_cnt[wib][lane] = 0u;
            __syncwarp();
            if (__any_sync(full, active)) {
                const EdgeUV uv = edge_uv(frame, P, Q);
                // rows of the group's window, and its box
                int ylo = 0x7fffffff, yhi = -1;
                float bx0 = INFINITY, by0 = INFINITY, bx1 = -INFINITY, by1 = -INFINITY;
                if (active) {
                    const float lo = floorf(fminf(uv.v0, uv.v1) - uv.m) - 1.f;
                    const float hi = floorf(fmaxf(uv.v0, uv.v1) + uv.m) + 1.f;
                    ylo = lo > 0.f ? (int)fminf(lo, 2e9f) : 0;
                    yhi = hi < (float)(O.dimy - 1) ? (int)hi : O.dimy - 1;
                    bx0 = fminf(P.x, Q.x);
                    bx1 = fmaxf(P.x, Q.x);
                    by0 = fminf(P.y, Q.y);
                    by1 = fmaxf(P.y, Q.y);
                }
                ylo = __reduce_min_sync(full, ylo);
                yhi = __reduce_max_sync(full, yhi);
                for (int o = 16; o; o >>= 1) {
                    bx0 = fminf(bx0, __shfl_xor_sync(full, bx0, o));
                    by0 = fminf(by0, __shfl_xor_sync(full, by0, o));
                    bx1 = fmaxf(bx1, __shfl_xor_sync(full, bx1, o));
                    by1 = fmaxf(by1, __shfl_xor_sync(full, by1, o));
                }
                const Group grp{&O, mr, b0, R, ylo};
                // FP32 rejection: margins of 1e-6 (~17 u32) times the largest
                // products a vertex of O can give
                const float ex = Q.x - P.x, ey = Q.y - P.y;
                const float ru = fmaxf(fabsf((float)O.mbr[0] - P.x), fabsf((float)O.mbr[2] - P.x));
                const float rv = fmaxf(fabsf((float)O.mbr[1] - P.y), fabsf((float)O.mbr[3] - P.y));
                const float ma = 1.1e-6f * (fabsf(ex) * rv + fabsf(ey) * ru);
                const float rm = 1.1e-6f * (ru + rv + fabsf(ex) + fabsf(ey));
                // Rows, a row's BORDER pixels 32 at a time, their sequences 32 at a
                // time, and these' edges 32 at a time, as one loop: each step takes
                // the innermost that is left, and what is queued is worked off in
                // one place (the kernel's code is larger than the instruction cache
                // takes lightly; with a copy per use 40% of the stalls were on it).
                int ln = 0, qn = 0, hn = 0;
                uint32_t step = 0, turn = share->own;
                int y = ylo - 1, x0 = 0;
                int2 col = make_int2(0, -1);
                uint32_t s0 = 0, tsq = 0, k0 = 0, te = 0;
                uint32_t pid = 0, sq0 = 0, xsq = 0, qq = 0, qpid = 0, xe = 0;
                uint2 sq = make_uint2(0u, 0u);
#pragma unroll 1
                for (bool end = false; !end;) {
                    bool look_all = false;
                    if (k0 < te) {
                        const uint32_t k = k0 + lane;
                        k0 += 32;
                        const int oe = warp_owner(xe, k);
                        const uint32_t f = __shfl_sync(full, sq.x, oe) + (k - __shfl_sync(full, xe, oe));
                        const uint32_t fq = __shfl_sync(full, qq, oe), fpid = __shfl_sync(full, qpid, oe);
                        bool in = false;
                        if (k < te) {
                            const float2 A = orr[f], B = orr[f + 1];
                            in = !(fmaxf(A.x, B.x) < bx0 || fminf(A.x, B.x) > bx1 || fmaxf(A.y, B.y) < by0 ||
                                   fminf(A.y, B.y) > by1);
                        }
                        const unsigned m = __ballot_sync(full, in);
                        if (in) list[ln + __popc(m & ((1u << lane) - 1u))] = AreaListing{f, fpid, fq, col.x};
                        ln += __popc(m);
                        if (ln < 32) continue;
                    } else if (s0 < tsq && step == limit &&
                               area_spill(a.pool, share, it, state,
                                          (float)step / (float)(y - ylo + 1) * (float)(yhi - y + 1), lane)) {
                        end = look_all = true;
                    } else if (s0 < tsq) {
                        const uint32_t si = s0 + lane;
                        s0 += 32;
                        if (step++ != turn) continue;
                        turn += share->stride;
                        const int ow = warp_owner(xsq, si);
                        qq = __shfl_sync(full, sq0, ow) + (si - __shfl_sync(full, xsq, ow));
                        qpid = __shfl_sync(full, pid, ow);
                        sq = si < tsq ? oseq[qq] : make_uint2(0u, 0u);
                        xe = warp_excl_scan(sq.y, lane, te);
                        k0 = 0;
                        continue;
                    } else if (x0 <= col.y) {
                        const int x = x0 + lane;
                        x0 += 32;
                        pid = (uint32_t)(y * O.dimx + x);
                        sq0 = 0;
                        uint32_t nsq = 0;
                        if (x <= col.y && show_status(ost[pid], cc) == 1) {
                            sq0 = ooff[pid];
                            nsq = ooff[pid + 1] - sq0;
                        }
                        xsq = warp_excl_scan(nsq, lane, tsq);
                        s0 = 0;
                        continue;
                    } else {
                        // a listing is looked up from its own row, so it may not
                        // wait while the ring of kept rows moves on
                        end = ++y > yhi;
                        look_all = end || ((y - ylo) & (kQueueRows - 1)) == 0;
                        if (!end) {
                            col = active ? edge_columns(uv, y, O.dimx) : make_int2(0x7fffffff, -1);
                            col.x = __reduce_min_sync(full, col.x);
                            col.y = __reduce_max_sync(full, col.y);
                            x0 = col.x;
                            if (lane == 0) rows[y & (kRowCache - 1)] = col;
                            if (!look_all || !ln) continue;
                        }
                    }
                    __syncwarp();
                    // 32 listings, or all: those that are their edge's first go on
                    if (ln >= 32 || (look_all && ln)) {
                        uint32_t f = 0;
                        bool keep = false;
                        if (lane < ln) {
                            const AreaListing l = list[lane];
                            f = l.f;
                            keep = first_listing(sv, grp, rows, a.ep_off, a.ep_pix, cc, l.pid, l.lo, l.q, f);
                        }
                        const unsigned kept = __ballot_sync(full, keep);
                        if (keep) {
                            const int at = qn + __popc(kept & ((1u << lane) - 1u));
                            const float2 A = orr[f], B = orr[f + 1];
                            seg[at] = make_float4(A.x, A.y, B.x, B.y);
                            edge[at] = f;
                        }
                        qn += __popc(kept);
                        ln = max(ln - 32, 0);
                        AreaListing mv{};
                        if (lane < ln) mv = list[32 + lane];
                        __syncwarp();
                        if (lane < ln) list[lane] = mv;
                        __syncwarp();
                    }
                    // 32 edges, at the end all, against every lane's edge; and 32
                    // pairs that may cross, at the end all, in FP64, one per lane
                    while (qn >= 32 || (end && (qn | hn))) {
                        const int m = min(qn, 32);
                        unsigned hits = 0, known = 0;  // known: both ends clearly on either side, of both
                        if (active) {
#pragma unroll 1
                            for (int j = (int)slice; j < m; j += (int)G) {
                                const float4 s = seg[j];
                                const float U = s.x - P.x, V = s.y - P.y, U2 = s.z - P.x, V2 = s.w - P.y;
                                const float oc = __fmaf_rn(ex, V, -(ey * U)), od = __fmaf_rn(ex, V2, -(ey * U2));
                                const float gx = U2 - U, gy = V2 - V;
                                const float op = __fmaf_rn(gy, U, -(gx * V));
                                const float oq = op + __fmaf_rn(gx, ey, -(gy * ex));
                                const float mb = rm * (fabsf(gx) + fabsf(gy));
                                if (!(fminf(oc, od) > ma || fmaxf(oc, od) < -ma || fminf(op, oq) > mb ||
                                      fmaxf(op, oq) < -mb))
                                    hits |= 1u << j;
                                if (fminf(oc, od) < -ma && fmaxf(oc, od) > ma && fminf(op, oq) < -mb &&
                                    fmaxf(op, oq) > mb)
                                    known |= 1u << j;
                            }
                        }
                        const int left = qn - m;
                        unsigned any;
                        do {
                            any = __ballot_sync(full, hits != 0);
                            if (hits) {
                                const int at = hn + __popc(any & ((1u << lane) - 1u));
                                const int j = __ffs(hits) - 1;
                                hit[at] = edge[j];
                                hedge[at] = (uint8_t)((uint32_t)lane % R | (known >> j & 1u) << 5);
                                hits &= hits - 1;
                            }
                            hn += __popc(any);
                            if (hn >= 32 || (end && !left && !any && hn)) {
                                __syncwarp();
                                if (lane < hn) {
                                    const uint32_t h = hedge[lane], k = h & 31u, f = hit[lane];
                                    const float2 A = mr[b0 + k], B = mr[b0 + k + 1];
                                    double t, den;
                                    my_tests++;
                                    if (crossing(A, B, orr, f, (h & 32u) != 0, t, den)) {
                                        const long long v = __double2ll_rn(t * kParamScale);
                                        const unsigned long long w = (unsigned long long)((den > 0) == inner_left ? v : -v);
                                        const uint32_t wl = (uint32_t)w;
                                        const uint32_t old = atomicAdd(&s_lo[wib][k], wl);
                                        atomicAdd(&s_hi[wib][k], (uint32_t)(w >> 32) + (old + wl < wl ? 1u : 0u));
                                        atomicAdd(&s_cnt[wib][k], 1u);
                                    }
                                }
                                hn = max(hn - 32, 0);
                                uint32_t mv = 0;
                                uint8_t mk = 0;
                                if (lane < hn) {
                                    mv = hit[32 + lane];
                                    mk = hedge[32 + lane];
                                }
                                __syncwarp();
                                if (lane < hn) {
                                    hit[lane] = mv;
                                    hedge[lane] = mk;
                                }
                            }
                        } while (any);
                        qn = left;
                        float4 mv = make_float4(0.f, 0.f, 0.f, 0.f);
                        uint32_t mf = 0;
                        if (lane < qn) {
                            mv = seg[32 + lane];
                            mf = edge[32 + lane];
                        }
                        __syncwarp();
                        if (lane < qn) {
                            seg[lane] = mv;
                            edge[lane] = mf;
                        }
                        __syncwarp();
                    }
                }
            }
            __syncwarp();
            if (AreaSpill *sp = share->sp) {
                // its sums to the pool; the last part takes all of them
                const unsigned long long v = (unsigned long long)s_hi[wib][lane] << 32 | s_lo[wib][lane];
                if (share->left) {
                    sp->sum[lane] = v;
                    sp->cnt[lane] = s_cnt[wib][lane];
                    continue;
                }
                if (s_cnt[wib][lane]) {
                    atomicAdd(&sp->sum[lane], v);
                    atomicAdd(&sp->cnt[lane], s_cnt[wib][lane]);
                }
                __threadfence();
                __syncwarp();
                if (lane == 0) share->left = atomicAdd(&sp->done, 1u) + 1u != share->stride;
                __syncwarp();
                if (share->left) continue;
                __threadfence();
                const unsigned long long tot = __ldcg(&sp->sum[lane]);
                s_lo[wib][lane] = (uint32_t)tot;
                s_hi[wib][lane] = (uint32_t)(tot >> 32);
                s_cnt[wib][lane] = __ldcg(&sp->cnt[lane]);
                __syncwarp();
            }
            // parity of crossings of earlier edges of the chunk
            const bool valid = (uint32_t)lane < R;
            const uint32_t tot_c = valid ? s_cnt[wib][lane] : 0u;
            const unsigned odd = __ballot_sync(full, valid && (tot_c & 1));
            const bool s_here = state ^ (__popc(odd & ((1u << lane) - 1)) & 1);
            const long long tail = (s_here ^ (tot_c & 1)) ? 1ll << 60 : 0ll;
            const long long inside =
                valid ? (long long)((unsigned long long)s_hi[wib][lane] << 32 | s_lo[wib][lane]) + tail : 0ll;
            const float z = (P.x - P.x) + (P.y - P.y) + (Q.x - Q.x) + (Q.y - Q.y);  // NaN unless they are finite
            if (__any_sync(full, inside != 0 || z != 0.f)) {  // a group outside adds nothing
                const double px = (double)P.x - ox, py = (double)P.y - oy;
                const double dx = (double)Q.x - P.x, dy = (double)Q.y - P.y;
                if (valid) acc += cross2(px, py, dx, dy) * ((double)inside * (1.0 / kParamScale));
            }
            my_cross += (unsigned long long)tot_c;
            state ^= (__popc(odd) & 1);
            __syncwarp();
        }
        if (share->left) continue;
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(full, acc, o);
        if (lane == 0) a.partial[it] = 0.5 * sign * acc;
    }
    if (my_tests) atomicAdd(&a.work[0], my_tests);
    if (my_cross) atomicAdd(&a.work[1], my_cross);
}

// orientation sign of every polygon (shoelace about its first vertex)
__global__ void k_orient(const StoreView sv, uint32_t npoly, int8_t *__restrict__ out) {
    const int lane = threadIdx.x & 31;
    uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t p = w; p < npoly; p += nw) {
        const PolyHdr &h = sv.hdr[p];
        const float2 *r = sv.ring + h.ring;
        double ox = r[0].x, oy = r[0].y, sa = 0;
        for (uint32_t k = lane; k + 1 < h.nv; k += 32)
            sa += cross2((double)r[k].x - ox, (double)r[k].y - oy, (double)r[k + 1].x - ox, (double)r[k + 1].y - oy);
        for (int o = 16; o; o >>= 1) sa += __shfl_xor_sync(0xffffffffu, sa, o);
        if (lane == 0) out[p] = sa >= 0 ? 1 : -1;
    }
}

// Edge -> pixel index of every rasterized polygon, by ring position: pass 0
// counts the pixels listing each edge, pass 1 writes them (in any order). A
// block per polygon, its warps over the pixels 32 at a time; these' sequences
// and their edges are flattened over the lanes, so that the atomics of a
// pixel's edges are in flight together: latency is all there is to it (1,440
// polygons of up to 1,024 vertices: 47 and 185 us a pass with a lane per pixel
// and a warp per polygon).
constexpr int kEdgePixWarps = 4;
template <bool kFill>
__global__ void __launch_bounds__(32 * kEdgePixWarps) k_edge_pix(const StoreView sv, uint32_t npoly,
                                                                 const uint64_t *__restrict__ ep_off,
                                                                 unsigned long long *__restrict__ cnt,
                                                                 uint32_t *__restrict__ ep_pix) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    for (uint32_t p = blockIdx.x; p < npoly; p += gridDim.x) {
        const PolyHdr &h = sv.hdr[p];
        if (h.err) continue;
        const uint32_t *off = sv.offset + h.off;
        const uint2 *seq = sv.seq + h.seq;
        for (uint32_t p0 = threadIdx.x & ~31u; p0 < h.P; p0 += blockDim.x) {
            const uint32_t pid = p0 + lane;
            const uint32_t q0 = pid < h.P ? off[pid] : 0u, nq = pid < h.P ? off[pid + 1] - q0 : 0u;
            uint32_t tsq;
            const uint32_t xsq = warp_excl_scan(nq, lane, tsq);
            for (uint32_t s0 = 0; s0 < tsq; s0 += 32) {
                const uint32_t si = s0 + lane;
                const int ow = warp_owner(xsq, si);
                const uint32_t q = __shfl_sync(full, q0, ow) + (si - __shfl_sync(full, xsq, ow));
                const uint32_t qpid = __shfl_sync(full, pid, ow);
                const uint2 sq = si < tsq ? seq[q] : make_uint2(0u, 0u);
                uint32_t te;
                const uint32_t xe = warp_excl_scan(sq.y, lane, te);
                for (uint32_t k0 = 0; k0 < te; k0 += 32) {
                    const uint32_t k = k0 + lane;
                    const int oe = warp_owner(xe, k);
                    const uint32_t f = __shfl_sync(full, sq.x, oe) + (k - __shfl_sync(full, xe, oe));
                    const uint32_t fpid = __shfl_sync(full, qpid, oe);
                    if (k >= te || f > h.nv) continue;  // past the polygon's ring slots (never, by construction)
                    const uint64_t g = h.ring + f;
                    const unsigned long long at = atomicAdd(&cnt[g], 1ull);
                    if (kFill) ep_pix[ep_off[g] + at] = fpid;
                }
            }
        }
    }
}

// Each edge's pixel list in ascending pixel id (insertion sort: an edge is
// listed by at most dimx + dimy pixels, a few in the common case).
__global__ void k_edge_pix_sort(const uint64_t *__restrict__ ep_off, uint64_t nring, uint32_t *__restrict__ ep_pix) {
    for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < nring; g += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t b = ep_off[g], e = ep_off[g + 1];
        for (uint64_t i = b + 1; i < e; i++) {
            const uint32_t v = ep_pix[i];
            uint64_t j = i;
            while (j > b && ep_pix[j - 1] > v) {
                ep_pix[j] = ep_pix[j - 1];
                j--;
            }
            ep_pix[j] = v;
        }
    }
}

// items per pair, for every slot up to cap (0 past the pair count)
__global__ void k_area_items(const StoreView sv, const uint32_t *__restrict__ pairs, const uint64_t *__restrict__ np,
                             uint64_t cap, uint64_t tgt_base, Chunks chunks, uint64_t *__restrict__ cnt) {
    const uint64_t n = *np;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k <= cap; k += (uint64_t)gridDim.x * blockDim.x) {
        if (k >= n) {
            cnt[k] = 0;
            continue;
        }
        const PolyHdr &S = sv.hdr[pairs[2 * k]];
        const PolyHdr &T = sv.hdr[tgt_base + pairs[2 * k + 1]];
        if (S.err || T.err) {
            cnt[k] = 0;
            continue;
        }
        uint32_t es = S.nv - 1, et = T.nv - 1;
        const uint32_t chunk = chunks.of(es, et);
        cnt[k] = (es + chunk - 1) / chunk + (et + chunk - 1) / chunk;
    }
}

// fixed-order sum of each pair's item partials
__global__ void k_area_reduce(const uint64_t *__restrict__ item_start, const uint64_t *__restrict__ np,
                              const double *__restrict__ partial, const StoreView sv,
                              const uint32_t *__restrict__ pairs, uint64_t tgt_base, double *__restrict__ out) {
    const uint64_t n = *np;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (uint64_t)gridDim.x * blockDim.x) {
        const PolyHdr &S = sv.hdr[pairs[2 * k]];
        const PolyHdr &T = sv.hdr[tgt_base + pairs[2 * k + 1]];
        if (S.err || T.err) {
            out[k] = nan("");
            continue;
        }
        double s = 0;
        for (uint64_t i = item_start[k]; i < item_start[k + 1]; i++) s += partial[i];
        out[k] = fabs(s);
    }
}

// ---------------------------------------------------------------- host --

static Chunks chunks_of(const farm_store *s) {
    Chunks c;
    for (int b = 0; b < 32; b++) c.c[b] = (uint16_t)(s->area_chunk[b] > 0 ? s->area_chunk[b] : kDefaultChunk);
    return c;
}

// polygon orientations, computed once per rasterization, in a scratch slot of
// their own (a captured plan holds its address)
constexpr int kOrientSlot = Q_AREA_ORIENT;
static int ensure_orient(farm_store *s, cudaStream_t st) {
    DevBuf &ori = s->s[kOrientSlot];
    if (s->orient_epoch == s->raster_epoch && ori.cap >= s->n_poly) return FARM_OK;
    FARM_TRY(ori.ensure(s->n_poly + 64));
    unsigned ob = (unsigned)((32ull * s->n_poly + 255) / 256);
    if (ob > 8192) ob = 8192;
    k_orient<<<ob, 256, 0, st>>>(s->view(), (uint32_t)s->n_poly, ori.as<int8_t>());
    s->launches++;
    FARM_CUDA(cudaGetLastError());
    s->orient_epoch = s->raster_epoch;
    return FARM_OK;
}

// The edge -> pixel index, built once per rasterization in scratch slots of
// its own (a captured plan holds their addresses). Counts go through Q_SCR3.
static int ensure_edge_pix(farm_store *s, cudaStream_t st) {
    if (s->edgepix_epoch == s->raster_epoch) return FARM_OK;
    const uint64_t nring = s->n_edges + 2 * s->n_poly;
    DevBuf &off = s->s[Q_AREA_EPOFF], &pix = s->s[Q_AREA_EPPIX], &cnt = s->s[Q_SCR3];
    FARM_TRY(off.ensure(8 * (nring + 1) + 64));
    FARM_TRY(cnt.ensure(8 * (nring + 1) + 64));
    unsigned long long *c = cnt.as<unsigned long long>();
    uint64_t *o = off.as<uint64_t>();
    const unsigned blocks = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(s->n_poly, 16384));
    FARM_CUDA(cudaMemsetAsync(c, 0, 8 * (nring + 1), st));
    k_edge_pix<false><<<blocks, 32 * kEdgePixWarps, 0, st>>>(s->view(), (uint32_t)s->n_poly, nullptr, c, nullptr);
    FARM_CUDA(cudaGetLastError());
    size_t bytes = 0;
    FARM_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, bytes, (const uint64_t *)c, o, (int64_t)(nring + 1)));
    FARM_TRY(s->cub_tmp.ensure(bytes + 64));
    FARM_CUDA(cub::DeviceScan::ExclusiveSum(s->cub_tmp.p, bytes, (const uint64_t *)c, o, (int64_t)(nring + 1), st));
    uint64_t total = 0;
    FARM_CUDA(cudaMemcpyAsync(&total, o + nring, 8, cudaMemcpyDeviceToHost, st));
    FARM_CUDA(cudaStreamSynchronize(st));
    FARM_TRY(pix.ensure(4 * total + 64));
    FARM_CUDA(cudaMemsetAsync(c, 0, 8 * (nring + 1), st));
    k_edge_pix<true><<<blocks, 32 * kEdgePixWarps, 0, st>>>(s->view(), (uint32_t)s->n_poly, o, c, pix.as<uint32_t>());
    FARM_CUDA(cudaGetLastError());
    unsigned sb = (unsigned)((nring + 255) / 256);
    if (sb > 8192) sb = 8192;
    k_edge_pix_sort<<<sb ? sb : 1, 256, 0, st>>>(o, nring, pix.as<uint32_t>());
    FARM_CUDA(cudaGetLastError());
    s->launches += 4;
    s->edgepix_epoch = s->raster_epoch;
    return FARM_OK;
}

// Buffers of one area pass. Everything the kernels need to know about the
// batch (pair count, item count) is read on the device, so the same sequence
// can be captured once in a CUDA graph and replayed for any batch that fits.
struct AreaBufs {
    const uint32_t *pairs;
    const uint64_t *n;  // device scalar
    uint64_t cap_pairs;
    uint64_t *cnt, *start;  // cap_pairs + 1 each
    double *partial;
    uint64_t cap_items;
    unsigned long long *ctr;  // [0] work counter, [1] [2] overflow flags
    void *scan_tmp;
    size_t scan_bytes;
    double *out;
    Chunks chunks;
    AreaPool pool;
};

// The pool's memory: a chunk per eight items (one in 14 of 801 pairs of up to
// 20,000 vertices is cut). Without it (an allocation that fails) every item
// stays with its warp.
static AreaPool area_pool(DevBuf &b, uint64_t items, unsigned long long *ctr) {
    AreaPool p;
    const uint64_t cap = std::min<uint64_t>(32768, std::max<uint64_t>(512, items / 8));
    if (b.ensure(cap * (sizeof(AreaSpill) + kAreaParts * sizeof(uint2)) + 64) != FARM_OK) return p;
    p.chunk = b.as<AreaSpill>();
    p.unit = reinterpret_cast<uint2 *>(p.chunk + cap);
    p.ctr = ctr;
    p.cap = (uint32_t)cap;
    return p;
}

static int scan_bytes(uint64_t cap, size_t *bytes) {
    FARM_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, *bytes, (const uint64_t *)nullptr, (uint64_t *)nullptr,
                                            (int64_t)(cap + 1)));
    return FARM_OK;
}

static int area_items(farm_store *s, const AreaBufs &b, cudaStream_t st) {
    unsigned blocks = (unsigned)((b.cap_pairs + 256) / 256);
    if (blocks > 4096) blocks = 4096;
    k_area_items<<<blocks, 256, 0, st>>>(s->view(), b.pairs, b.n, b.cap_pairs, s->n_side[0], b.chunks, b.cnt);
    FARM_CUDA(cudaGetLastError());
    size_t bytes = b.scan_bytes;
    FARM_CUDA(cub::DeviceScan::ExclusiveSum(b.scan_tmp, bytes, b.cnt, b.start, (int64_t)(b.cap_pairs + 1), st));
    return FARM_OK;
}

static int area_compute(farm_store *s, const AreaBufs &b, cudaStream_t st) {
    FARM_CUDA(cudaMemsetAsync(b.ctr, 0, 64, st));
    AreaArgs aa{b.pairs,
                b.n,
                s->n_side[0],
                b.chunks,
                b.start,
                b.cap_items,
                b.partial,
                s->s[kOrientSlot].as<int8_t>(),
                s->s[Q_AREA_EPOFF].as<uint64_t>(),
                s->s[Q_AREA_EPPIX].as<uint32_t>(),
                b.ctr,
                b.ctr + 1,
                b.ctr + 3,
                spread_items(),
                b.pool,
                0};
    k_area<<<sm_count() * 8, 256, 0, st>>>(s->view(), aa);
    FARM_CUDA(cudaGetLastError());
    if (b.pool.cap) {
        aa.rest = 1;
        k_area<<<sm_count() * 3, 256, 0, st>>>(s->view(), aa);
        FARM_CUDA(cudaGetLastError());
    }
    unsigned blocks = (unsigned)((b.cap_pairs + 255) / 256);
    if (blocks > 4096) blocks = 4096;
    if (!blocks) blocks = 1;
    k_area_reduce<<<blocks, 256, 0, st>>>(b.start, b.n, b.partial, s->view(), b.pairs, s->n_side[0], b.out);
    FARM_CUDA(cudaGetLastError());
    return FARM_OK;
}

static int area_checks(farm_store *s, const char *who) {
    if (!s->rasterized) {
        set_error(std::string(who) + ": rasterize first");
        return FARM_EINVAL;
    }
    if (s->n_side[1] == 0) {
        set_error(std::string(who) + ": no target side loaded");
        return FARM_EINVAL;
    }
    return FARM_OK;
}

int intersection_area(farm_store *s, const uint32_t *pairs, uint64_t n, int mem, double *out, farm_stats *st) {
    FARM_TRY(area_checks(s, "farm_intersection_area"));
    FARM_TRY(check_pairs(s, pairs, n, mem, false, "farm_intersection_area"));
    cudaStream_t stream = s->stream;
    const uint32_t *dpairs = pairs;
    if (mem == FARM_MEM_HOST && n) {
        FARM_TRY(s->d_pairs.ensure(8 * n));
        FARM_CUDA(cudaMemcpyAsync(s->d_pairs.p, pairs, 8 * n, cudaMemcpyHostToDevice, stream));
        dpairs = s->d_pairs.as<uint32_t>();
    }
    double *dout = out;
    if (mem == FARM_MEM_HOST || !out) {
        FARM_TRY(s->d_out.ensure(8 * n + 64));
        dout = s->d_out.as<double>();
    }
    DevBuf &cnt = s->s[Q_SCR0], &start = s->s[Q_SCR1], &part = s->s[Q_SCR2];
    FARM_TRY(cnt.ensure(8 * (n + 1) + 64));
    FARM_TRY(start.ensure(8 * (n + 1) + 64));
    FARM_TRY(s->d_counters.ensure(256));
    unsigned long long *ctr = s->d_counters.as<unsigned long long>();
    uint64_t *dn = reinterpret_cast<uint64_t *>(ctr + 8);
    FARM_CUDA(cudaMemcpyAsync(dn, &n, 8, cudaMemcpyHostToDevice, stream));
    FARM_TRY(ensure_orient(s, stream));
    FARM_TRY(ensure_edge_pix(s, stream));
    AreaBufs b{};
    b.pairs = dpairs;
    b.n = dn;
    b.cap_pairs = n;
    b.cnt = cnt.as<uint64_t>();
    b.start = start.as<uint64_t>();
    b.ctr = ctr;
    b.out = dout;
    b.chunks = chunks_of(s);
    FARM_TRY(scan_bytes(n, &b.scan_bytes));
    FARM_TRY(s->cub_tmp.ensure(b.scan_bytes + 64));
    b.scan_tmp = s->cub_tmp.p;
    FARM_CUDA(cudaEventRecord(s->ev[6], stream));
    FARM_TRY(area_items(s, b, stream));
    uint64_t nitems = 0;
    FARM_CUDA(cudaMemcpyAsync(&nitems, b.start + n, 8, cudaMemcpyDeviceToHost, stream));
    FARM_CUDA(cudaStreamSynchronize(stream));
    FARM_TRY(part.ensure(8 * nitems + 64));
    b.partial = part.as<double>();
    b.pool = area_pool(s->s[Q_SPILL], nitems, ctr + 5);
    b.cap_items = nitems;
    FARM_TRY(area_compute(s, b, stream));
    FARM_CUDA(cudaEventRecord(s->ev[7], stream));
    if (mem == FARM_MEM_HOST && out && n) FARM_CUDA(cudaMemcpyAsync(out, dout, 8 * n, cudaMemcpyDeviceToHost, stream));
    unsigned long long work[2] = {0, 0};
    FARM_CUDA(cudaMemcpyAsync(work, ctr + 3, 16, cudaMemcpyDeviceToHost, stream));
    FARM_CUDA(cudaStreamSynchronize(stream));
    s->launches += b.pool.cap ? 5 : 4;
    if (st) {
        memset(st, 0, sizeof *st);
        st->pairs = n;
        st->segment_tests = work[0];
        st->border_pairs = work[1];
        float ms = 0;
        cudaEventElapsedTime(&ms, s->ev[6], s->ev[7]);
        st->ms_total = ms;
        st->ms_stage[2] = ms;
        st->kernel_launches = b.pool.cap ? 5 : 4;
    }
    return FARM_OK;
}

}  // namespace farm

extern "C" int farm_intersection_area(farm_store *s, const uint32_t *pairs, uint64_t n, int mem, double *out,
                                      farm_stats *st) {
    using namespace farm;
    if (!s || (n && !pairs)) {
        set_error("invalid arguments to farm_intersection_area");
        return FARM_EINVAL;
    }
    return intersection_area(s, pairs, n, mem, out, st);
}

// ------------------------------------------------------ plans and tuning --
// A plan owns fixed-capacity buffers for one area pass and the CUDA graph of
// that pass (items, scan, the persistent work-stealing kernel, the per-pair
// reduction), captured once. Running it copies a batch of pairs in and
// replays the graph: one launch for any batch within capacity, whatever its
// mix of tiny and huge pairs.
struct farm_area_plan {
    farm_store *s = nullptr;
    uint64_t cap_pairs = 0, cap_items = 0, epoch = 0;
    farm::DevBuf pairs, n, cnt, start, partial, ctr, tmp, out, pool;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
};

namespace {
void plan_free(farm_area_plan *p) {
    if (!p) return;
    if (p->exec) cudaGraphExecDestroy(p->exec);
    if (p->graph) cudaGraphDestroy(p->graph);
    for (farm::DevBuf *b : {&p->pairs, &p->n, &p->cnt, &p->start, &p->partial, &p->ctr, &p->tmp, &p->out, &p->pool})
        b->release();
    delete p;
}
}  // namespace

extern "C" int farm_area_plan_create(farm_store *s, uint64_t max_pairs, uint64_t max_items, farm_area_plan **out) {
    using namespace farm;
    if (!s || !out || max_pairs == 0 || max_items == 0) {
        set_error("invalid arguments to farm_area_plan_create");
        return FARM_EINVAL;
    }
    *out = nullptr;
    FARM_TRY(area_checks(s, "farm_area_plan_create"));
    cudaStream_t st = s->stream;
    FARM_TRY(ensure_orient(s, st));
    FARM_TRY(ensure_edge_pix(s, st));
    farm_area_plan *p = new farm_area_plan();
    p->s = s;
    p->cap_pairs = max_pairs;
    p->cap_items = max_items;
    p->epoch = s->raster_epoch;
    AreaBufs b{};
    int rc = FARM_OK;
    if (rc == FARM_OK) rc = p->pairs.ensure(8 * max_pairs + 64);
    if (rc == FARM_OK) rc = p->n.ensure(64);
    if (rc == FARM_OK) rc = p->cnt.ensure(8 * (max_pairs + 1) + 64);
    if (rc == FARM_OK) rc = p->start.ensure(8 * (max_pairs + 1) + 64);
    if (rc == FARM_OK) rc = p->partial.ensure(8 * max_items + 64);
    if (rc == FARM_OK) rc = p->ctr.ensure(128);
    if (rc == FARM_OK) rc = p->out.ensure(8 * max_pairs + 64);
    if (rc == FARM_OK) rc = scan_bytes(max_pairs, &b.scan_bytes);
    if (rc == FARM_OK) rc = p->tmp.ensure(b.scan_bytes + 64);
    if (rc == FARM_OK) {
        cudaError_t e = cudaMemsetAsync(p->n.p, 0, 8, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (e != cudaSuccess) rc = cuda_fail(e, "farm_area_plan_create");
    }
    if (rc != FARM_OK) {
        plan_free(p);
        return rc;
    }
    b.pairs = p->pairs.as<uint32_t>();
    b.n = p->n.as<uint64_t>();
    b.cap_pairs = max_pairs;
    b.cnt = p->cnt.as<uint64_t>();
    b.start = p->start.as<uint64_t>();
    b.partial = p->partial.as<double>();
    b.cap_items = max_items;
    b.ctr = p->ctr.as<unsigned long long>();
    b.scan_tmp = p->tmp.p;
    b.out = p->out.as<double>();
    b.chunks = chunks_of(s);
    b.pool = area_pool(p->pool, max_items, b.ctr + 5);
    cudaError_t e = cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) {
        plan_free(p);
        return cuda_fail(e, "cudaStreamBeginCapture");
    }
    int rc1 = area_items(s, b, st);
    int rc2 = rc1 == FARM_OK ? area_compute(s, b, st) : rc1;
    e = cudaStreamEndCapture(st, &p->graph);
    if (rc2 != FARM_OK || e != cudaSuccess) {
        plan_free(p);
        return rc2 != FARM_OK ? rc2 : cuda_fail(e, "cudaStreamEndCapture");
    }
    e = cudaGraphInstantiate(&p->exec, p->graph, 0);
    if (e != cudaSuccess) {
        plan_free(p);
        return cuda_fail(e, "cudaGraphInstantiate");
    }
    *out = p;
    return FARM_OK;
}

extern "C" int farm_area_plan_run(farm_area_plan *p, const uint32_t *pairs, uint64_t n, int mem, double *out,
                                  farm_stats *st_out) {
    using namespace farm;
    if (!p || (n && (!pairs || !out))) {
        set_error("invalid arguments to farm_area_plan_run");
        return FARM_EINVAL;
    }
    farm_store *s = p->s;
    if (n > p->cap_pairs) {
        set_error("farm_area_plan_run: " + std::to_string(n) + " pairs exceed the plan's capacity of " +
                  std::to_string(p->cap_pairs));
        return FARM_EINVAL;
    }
    if (s->raster_epoch != p->epoch) {
        set_error("farm_area_plan_run: the store was reloaded or rasterized again since the plan was made");
        return FARM_EINVAL;
    }
    FARM_TRY(check_pairs(s, pairs, n, mem, false, "farm_area_plan_run"));
    cudaStream_t st = s->stream;
    const cudaMemcpyKind k_in = mem == FARM_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
    const cudaMemcpyKind k_out = mem == FARM_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
    if (n) FARM_CUDA(cudaMemcpyAsync(p->pairs.p, pairs, 8 * n, k_in, st));
    FARM_CUDA(cudaMemcpyAsync(p->n.p, &n, 8, cudaMemcpyHostToDevice, st));
    FARM_CUDA(cudaEventRecord(s->ev[6], st));
    FARM_CUDA(cudaGraphLaunch(p->exec, st));
    FARM_CUDA(cudaEventRecord(s->ev[7], st));
    unsigned long long flags[5] = {0, 0, 0, 0, 0};  // next, -, overflow, crossing tests, crossings
    FARM_CUDA(cudaMemcpyAsync(flags, p->ctr.p, 40, cudaMemcpyDeviceToHost, st));
    if (n) FARM_CUDA(cudaMemcpyAsync(out, p->out.p, 8 * n, k_out, st));
    FARM_CUDA(cudaStreamSynchronize(st));
    s->launches += p->pool.cap ? 4 : 3;
    if (flags[2]) {
        set_error("farm_area_plan_run: the batch needs more work items than the plan's capacity of " +
                  std::to_string(p->cap_items));
        return FARM_EOVERFLOW;
    }
    if (st_out) {
        memset(st_out, 0, sizeof *st_out);
        st_out->pairs = n;
        float ms = 0;
        cudaEventElapsedTime(&ms, s->ev[6], s->ev[7]);
        st_out->ms_total = ms;
        st_out->ms_stage[2] = ms;
        st_out->kernel_launches = 1;  // one graph launch
        st_out->segment_tests = flags[3];
        st_out->border_pairs = flags[4];
    }
    return FARM_OK;
}

extern "C" void farm_area_plan_destroy(farm_area_plan *p) { plan_free(p); }

extern "C" int farm_area_set_chunks(farm_store *s, const int32_t *chunk_by_bucket) {
    using namespace farm;
    if (!s || !chunk_by_bucket) {
        set_error("invalid arguments to farm_area_set_chunks");
        return FARM_EINVAL;
    }
    for (int b = 0; b < 32; b++)
        if (chunk_by_bucket[b] < 0 || chunk_by_bucket[b] > 32768) {
            set_error("farm_area_set_chunks: chunk sizes must lie in 1..32768 (0 = default)");
            return FARM_EINVAL;
        }
    for (int b = 0; b < 32; b++) s->area_chunk[b] = chunk_by_bucket[b];
    return FARM_OK;
}

extern "C" int farm_area_set_wide(farm_store *s, const int32_t *wide_by_bucket) {
    using namespace farm;
    if (!s || !wide_by_bucket) {
        set_error("invalid arguments to farm_area_set_wide");
        return FARM_EINVAL;
    }
    for (int b = 0; b < 32; b++)
        if (wide_by_bucket[b] < 0 || wide_by_bucket[b] > 65535) {
            set_error("farm_area_set_wide: window sizes must lie in 1..65535 (0 = default)");
            return FARM_EINVAL;
        }
    for (int b = 0; b < 32; b++) s->area_wide[b] = wide_by_bucket[b];
    return FARM_OK;
}

// Autotuner: for every size bucket present in the sample (floor(log2) of a
// pair's larger edge count), time the area pass on up to 2048 of its pairs
// over the candidate chunk sizes 8..256 (edges per work item) and keep the
// fastest. One untimed pass per bucket warms up. The store keeps the table
// (farm_area_set_chunks); it is also returned, with the window table, which
// nothing reads any more (farm_area_set_wide), at its default.
extern "C" int farm_area_autotune(farm_store *s, const uint32_t *pairs, uint64_t n, int mem, int32_t *chunk_out,
                                  int32_t *wide_out) {
    using namespace farm;
    if (!s || (n && !pairs)) {
        set_error("invalid arguments to farm_area_autotune");
        return FARM_EINVAL;
    }
    FARM_TRY(area_checks(s, "farm_area_autotune"));
    FARM_TRY(check_pairs(s, pairs, n, mem, false, "farm_area_autotune"));
    std::vector<uint32_t> hp(2 * n);
    if (n) {
        if (mem == FARM_MEM_HOST) {
            memcpy(hp.data(), pairs, 8 * n);
        } else {
            FARM_CUDA(cudaMemcpyAsync(hp.data(), pairs, 8 * n, cudaMemcpyDeviceToHost, s->stream));
            FARM_CUDA(cudaStreamSynchronize(s->stream));
        }
    }
    auto edges = [&](int side, uint32_t k) -> uint32_t {
        const std::vector<uint64_t> &o = s->h_off[side];
        return (uint32_t)(o[k + 1] - o[k]);  // stored vertices = edges of the in-memory ring
    };
    std::vector<std::vector<uint32_t>> byb(32);
    for (uint64_t i = 0; i < n; i++) {
        if (hp[2 * i] >= s->n_side[0] || hp[2 * i + 1] >= s->n_side[1]) {
            set_error("farm_area_autotune: pair index out of range");
            return FARM_EINVAL;
        }
        const int b = Chunks::bucket(edges(0, hp[2 * i]), edges(1, hp[2 * i + 1]));
        if (byb[b].size() < 2 * 2048) {
            byb[b].push_back(hp[2 * i]);
            byb[b].push_back(hp[2 * i + 1]);
        }
    }
    static const int32_t kChunkCand[] = {8, 16, 32, 64, 128, 256};
    int32_t saved_c[32];
    memcpy(saved_c, s->area_chunk, sizeof saved_c);
    int32_t best_c[32], best_w[32];
    memcpy(best_c, s->area_chunk, sizeof best_c);
    memcpy(best_w, s->area_wide, sizeof best_w);
    // one pass of bucket b's pairs with chunk c everywhere
    auto timed = [&](int b, int32_t c, double *ms) -> int {
        for (int q = 0; q < 32; q++) s->area_chunk[q] = c;
        farm_stats stt;
        const int rc = intersection_area(s, byb[b].data(), byb[b].size() / 2, FARM_MEM_HOST, nullptr, &stt);
        *ms = stt.ms_total;
        return rc;
    };
    for (int b = 0; b < 32; b++) {
        if (byb[b].empty()) continue;
        double ms = 0, best_ms = 1e300;
        int rc = timed(b, kDefaultChunk, &ms);  // warm-up
        int32_t bc = kDefaultChunk;
        for (int32_t c : kChunkCand) {
            if (rc == FARM_OK) rc = timed(b, c, &ms);
            if (rc == FARM_OK && ms < best_ms) {
                best_ms = ms;
                bc = c;
            }
        }
        if (rc != FARM_OK) {
            memcpy(s->area_chunk, saved_c, sizeof saved_c);
            return rc;
        }
        best_c[b] = bc;
        best_w[b] = kDefaultWide;
    }
    memcpy(s->area_chunk, best_c, sizeof best_c);
    memcpy(s->area_wide, best_w, sizeof best_w);
    if (chunk_out) memcpy(chunk_out, best_c, sizeof best_c);
    if (wide_out) memcpy(wide_out, best_w, sizeof best_w);
    return FARM_OK;
}
