// Stages (b) + (c) for within-distance: hierarchical BORDER x BORDER descent,
// candidate ordering and border refinement with point-segment distances.
//
// Reference decision procedure (Ideal::within, Ideal.cpp:2475-2643):
//  * descend the two polygons' raster hierarchies together (the coarser side
//    advances); at each level the BORDER children of the queued pixels form
//    two sets, their cross product gives the smallest box max-distance (any
//    max-distance <= d decides "true") and keeps the pairs whose box distance
//    is <= d and below that smallest max-distance;
//  * at the finest level the kept pairs are ordered by (approximate distance,
//    low, high, ids) and refined in that order with the minimum point-segment
//    distance of their edge sequences; "true" once the running minimum is
//    below d, "false" once it is below every later pair's lower bound.
// Below the finest level the queue only matters through the two sets of
// pixels it holds (the children of its members), so each level here keeps
// two pixel sets instead of an explicit pair queue.
//
// The ordered refinement has an order-free form. Every candidate but the last
// in order is followed by one whose lower bound is at most d, so "false" can
// only be decided at the last candidate, after its first sequence pair: the
// answer is "true" iff some point-segment distance of some candidate before
// the last is below d, or one of the last candidate's first sequence pair (and
// further ones only while no distance so far was below 100000, the minimum's
// start value). So nothing is sorted, any warp may test any candidate, and a
// point-segment test only has to tell whether its FP64 distance is below d,
// which FP32 with an error bound decides for all but a few.
//
// Kernels: k_within (one warp per pair) descends, tests the finest level's
// candidates one after the other, and spills what is past its budget;
// k_within_spill tests those over all warps.
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "common.cuh"
#include "spill.cuh"

namespace farm {

// util.h:68 (float constants) and the 900-entry longitude table (util.h:73),
// regenerated on the host from its defining formula.
__constant__ float c_mean20[20];
__constant__ double c_deg_lon[900];
__constant__ float c_inv_deg_lon_f[900];  // 1 / c_deg_lon, rounded to float (FP32 first pass only)

static std::mutex g_tab_mu;
static bool g_tab_ready[64] = {};

static int ensure_tables(int dev) {
    std::lock_guard<std::mutex> lock(g_tab_mu);
    if (dev >= 0 && dev < 64 && g_tab_ready[dev]) return FARM_OK;
    const float mean20[20] = {0.0f,  0.7f,  0.62f, 0.55f, 0.52f, 0.45f, 0.42f, 0.4f,  0.38f, 0.34f,
                              0.31f, 0.28f, 0.25f, 0.22f, 0.18f, 0.15f, 0.1f,  0.05f, 0.0f,  0.0f};
    double deg[900];
    const double PI = 3.14159265;
    for (int i = 0; i < 900; i++) {
        double lat = i / 10.0;
        double v = 360.0 / (sin((90 - lat) * PI / 180) * 40076);
        char buf[64];
        snprintf(buf, sizeof buf, "%.6f", v);
        deg[i] = strtod(buf, nullptr);
    }
    FARM_CUDA(cudaMemcpyToSymbol(c_mean20, mean20, sizeof mean20));
    FARM_CUDA(cudaMemcpyToSymbol(c_deg_lon, deg, sizeof deg));
    float inv[900];
    for (int i = 0; i < 900; i++) inv[i] = (float)(1.0 / deg[i]);
    FARM_CUDA(cudaMemcpyToSymbol(c_inv_deg_lon_f, inv, sizeof inv));
    if (dev >= 0 && dev < 64) g_tab_ready[dev] = true;
    return FARM_OK;
}

__device__ __forceinline__ double deg_lon(double lat) {
    double a = fabs(lat);
    if (a == 90) a = 89.9;
    int idx = (int)(a * 10);
    if (idx < 0 || idx >= 900) idx = 899;  // the reference indexes past the table here
    return c_deg_lon[idx];
}
#define DEG_LAT (360.0 / 40076.0)

struct Box {
    double lo0, lo1, hi0, hi1;
};

__device__ __forceinline__ Box pixel_box(const LayerGeom &g, int id) {
    int x = id % g.dimx, y = id / g.dimx;
    Box b;
    b.lo0 = g.mbr[0] + x * g.step_x;
    b.lo1 = g.mbr[1] + y * g.step_y;
    b.hi0 = g.mbr[0] + (x + 1) * g.step_x;
    b.hi1 = g.mbr[1] + (y + 1) * g.step_y;
    return b;
}

// Box.cpp:90-118
__device__ __noinline__ double box_distance(const Box &a, const Box &t, bool geo) {
    if (!(t.lo0 > a.hi0 || t.hi0 < a.lo0 || t.lo1 > a.hi1 || t.hi1 < a.lo1)) return 0;
    double dx = 0, dy = 0;
    if (t.lo1 > a.hi1)
        dy = t.lo1 - a.hi1;
    else if (t.hi1 < a.lo1)
        dy = a.lo1 - t.hi1;
    if (t.lo0 > a.hi0)
        dx = t.lo0 - a.hi0;
    else if (t.hi0 < a.lo0)
        dx = a.lo0 - t.hi0;
    if (geo) {
        dy = dy / DEG_LAT;
        dx = dx / deg_lon(a.lo1);
    }
    return sqrt(dx * dx + dy * dy);
}

// Box.cpp:120-149: the corners become float points first, and the result is
// the largest of the 16 corner-to-corner distances. A corner pair's x
// difference depends only on the two corners' x choices and its y difference
// only on their y choices, so the 16 pairs are every combination of one of
// the 4 x differences with one of the 4 y differences. Every step of a
// distance — the float subtraction, the division by the degree scale, the
// square, the sum and sqrt — is monotone in |dx| and |dy| under
// round-to-nearest, so the largest distance is the one built from the
// largest |dx| and the largest |dy|: the same double, with 2 divisions and
// one sqrt instead of 32 and 16.
__device__ __forceinline__ float4 box_corners_f(const Box &a) {
    return make_float4((float)a.lo0, (float)a.lo1, (float)a.hi0, (float)a.hi1);
}

// the same from the boxes' float corners (box_corners_f) and a's lo1. Of a box
// lo <= hi, so the largest |x difference| is one of hi - lo either way.
__device__ __forceinline__ float2 corner_spans(const float4 &fa, const float4 &ft) {
    return make_float2(fmaxf(__fsub_rn(fa.z, ft.x), __fsub_rn(ft.z, fa.x)),
                       fmaxf(__fsub_rn(fa.w, ft.y), __fsub_rn(ft.w, fa.y)));
}
__device__ __noinline__ double box_max_distance_f(const float4 &fa, const float4 &ft, double a_lo1, bool geo) {
    const float2 m = corner_spans(fa, ft);
    double dx = m.x, dy = m.y;
    if (geo) {
        dy = dy / DEG_LAT;
        dx = dx / deg_lon(a_lo1);
    }
    return sqrt(dx * dx + dy * dy);
}

// geometry_computation.h:49-89
__device__ __noinline__ double pt_seg_dist(float2 p, float2 p1, float2 p2, bool geo) {
    double A = __fsub_rn(p.x, p1.x), B = __fsub_rn(p.y, p1.y);
    double C = __fsub_rn(p2.x, p1.x), D = __fsub_rn(p2.y, p1.y);
    double dot = A * C + B * D;
    double len_sq = C * C + D * D;
    double param = -1;
    if (len_sq != 0) param = dot / len_sq;
    double xx, yy;
    if (param < 0) {
        xx = p1.x;
        yy = p1.y;
    } else if (param > 1) {
        xx = p2.x;
        yy = p2.y;
    } else {
        xx = p1.x + param * C;
        yy = p1.y + param * D;
    }
    double dx = p.x - xx, dy = p.y - yy;
    if (geo) {
        dx = dx / deg_lon(p.y);
        dy = dy / DEG_LAT;
    }
    return sqrt(dx * dx + dy * dy);
}

// The FP32 screen of pt_seg_dist(...) < thr. It works relative to p1 (the
// reference's own float differences A, B, C, D and the projection parameter
// clamped to [0, 1]), so absolute coordinates never enter its rounding:
//   |d32 - d64| <= 22 u32 (M + L) S + 7 u32 d32 + 8 u64 (|p| + |p1| + M + L) S
// with M = |A| + |B|, L = |C| + |D|, S the geography scale (1 when planar).
// The first term covers the FP32 dot / reciprocal / parameter / projection
// rounding and the float roundings of the differences the reference keeps in
// double; the second the scaling and squares; the third the reference's own
// FP64 rounding (its projection is taken in absolute coordinates). The
// distance to a segment is 1-Lipschitz in the clamped parameter times the
// segment length, so branch flips at the clamp stay inside the bound. The
// constants below are about 3x wider, as c0 (the threshold, the third term
// over the pair's largest coordinate) and k1 (the first); the relative term
// is in the final comparison. A test that is not clearly at or past the
// threshold, nor clearly below it (c1), is evaluated in FP64, so the answer is
// pt_seg_dist's.
struct Near {
    double thr;
    float c0, c1, k1;
};
constexpr float kScaleGeo = 111.5f;  // no degree is longer: 40076 / 360 km

__device__ __forceinline__ Near near_of(const PolyHdr &S, const PolyHdr &T, double thr, bool geo) {
    double m = 0;
    for (int k = 0; k < 4; k++) m = fmax(m, fmax(fabs(S.mbr[k]), fabs(T.mbr[k])));
    const float sc = geo ? kScaleGeo : 1.f;
    Near w;
    // the running minimum of the reference starts at 100000: any test is below a larger threshold
    w.thr = thr > 100000.0 ? (double)INFINITY : thr;
    w.c0 = (float)w.thr * 1.000001f + 5e-14f * (float)m * sc;
    w.c1 = (float)w.thr * 0.999999f - 5e-14f * (float)m * sc;
    w.k1 = 4e-6f * sc;
    return w;
}

// Longitude scale of a point by its latitude's table entry: x the scale, y the
// largest step to a neighbouring entry (the index may differ from the FP64
// one at a boundary).
__device__ __forceinline__ float2 lon_entry(int idx) {
    const float s0 = c_inv_deg_lon_f[idx];
    const float s1 = c_inv_deg_lon_f[idx + 1 < 900 ? idx + 1 : 899], s2 = c_inv_deg_lon_f[idx > 0 ? idx - 1 : 0];
    return make_float2(s0, 1.001f * fmaxf(fabsf(s1 - s0), fabsf(s2 - s0)));
}
__device__ __forceinline__ int lat_index(float lat) {
    float a = fabsf(lat);
    if (a == 90.f) a = 89.9f;
    const int idx = (int)(a * 10.f);
    return idx < 0 || idx >= 900 ? 899 : idx;
}

struct Seg {
    float2 p1, p2;
    float C, D, inv, L;
};
__device__ __forceinline__ Seg make_seg(float2 p1, float2 p2) {
    Seg g;
    g.p1 = p1;
    g.p2 = p2;
    g.C = __fsub_rn(p2.x, p1.x);
    g.D = __fsub_rn(p2.y, p1.y);
    const float len = __fmaf_rn(g.C, g.C, __fmul_rn(g.D, g.D));
    g.inv = len != 0.f ? __frcp_rn(len) : 0.f;
    g.L = fabsf(g.C) + fabsf(g.D);
    return g;
}

// The FP32 screen: *may unless the distance is surely not below the threshold,
// *sure when it surely is; e: the point's longitude entry.
template <bool kGeo>
__device__ __forceinline__ void screen(float2 p, float2 e, const Seg &g, const Near &w, bool &may, bool &sure) {
    const float A = __fsub_rn(p.x, g.p1.x), B = __fsub_rn(p.y, g.p1.y);
    const float t = __saturatef(__fmul_rn(__fmaf_rn(A, g.C, __fmul_rn(B, g.D)), g.inv));
    float dx = __fmaf_rn(-t, g.C, A), dy = __fmaf_rn(-t, g.D, B);
    float err = __fmul_rn(w.k1, fabsf(A) + fabsf(B) + g.L);
    if (kGeo) {
        err = __fmaf_rn(fabsf(dx), e.y, err);
        dx = __fmul_rn(dx, e.x);
        dy = __fmul_rn(dy, (float)(40076.0 / 360.0));
    }
    const float d2 = __fmaf_rn(dx, dx, __fmul_rn(dy, dy)), up = w.c0 + err, dn = w.c1 - err;
    may |= !(d2 > up * up * 1.00001f);
    sure |= dn > 0.f && d2 * 1.00001f < dn * dn;
}

// One side of a candidate pixel pair: its pixel's edge sequences.
struct SeqSet {
    const uint2 *seq;
    const float2 *ring;
    uint32_t a, b;  // sequences [a, b)
};
__device__ __forceinline__ SeqSet seq_set(const StoreView &sv, const PolyHdr &h, uint32_t id) {
    const uint32_t *o = sv.offset + h.off;
    return {sv.seq + h.seq, sv.ring + h.ring, o[id], o[id + 1]};
}

// Sequences of fewer than 2 points are skipped, and a sequence (start, len)
// reads points [start, start + len) and the len - 1 segments between them
// (segment_to_segment_within_batch). Over all sequence pairs of a pixel pair
// that is every point of one side against every segment of the other.

// Points staged per warp and side: (x, y, longitude entry), and those of them
// that start a segment (to the next one).
constexpr uint32_t kWPts = 128;
struct WStage {
    float4 pt[2][kWPts];
    uint8_t seg[2][kWPts];
    uint32_t nseg[2];
};

// The next chunk of a side's points, sequence after sequence (those of fewer
// than 2 points skipped), into st->pt[side]: its length, 0 past the last.
// (*g, *at): the group of 32 sequences and the point in it; a chunk that ends
// inside a group is followed by one that starts with its last point.
template <bool kGeo>
__device__ __noinline__ uint32_t stage_points(const SeqSet &Q, WStage *st, int side, const float2 *tab, uint32_t *g, uint32_t *at,
                                 int lane) {
    const unsigned full = 0xffffffffu;
    for (; Q.a + *g < Q.b; *g += 32, *at = 0) {
        const uint32_t i = Q.a + *g + lane;
        const uint2 e = i < Q.b ? Q.seq[i] : make_uint2(0u, 0u);
        const uint32_t mine = e.y >= 2 ? e.y : 0u;
        uint32_t incl = mine;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(full, incl, o);
            if (lane >= o) incl += u;
        }
        const uint32_t total = __shfl_sync(full, incl, 31), excl = incl - mine;
        if (total == 0 || (*at && total - *at < 2)) continue;  // empty, or only the repeated point left
        const uint32_t n = min(kWPts, total - *at);
        uint32_t ns = 0;
        __syncwarp();
        for (uint32_t k0 = 0; k0 < n; k0 += 32) {
            const uint32_t k = k0 + lane, f = *at + k;
            int ow = 0;
            for (int b = 16; b; b >>= 1)
                if (__shfl_sync(full, excl, ow + b) <= f) ow += b;
            const uint32_t start = __shfl_sync(full, e.x, ow), ex = __shfl_sync(full, excl, ow),
                           len = __shfl_sync(full, mine, ow);
            bool starts = false;
            if (k < n) {
                const float2 p = Q.ring[start + (f - ex)];
                const float2 s = kGeo ? tab[lat_index(p.y)] : make_float2(1.f, 0.f);
                st->pt[side][k] = make_float4(p.x, p.y, s.x, s.y);
                starts = f - ex + 1 < len && k + 1 < n;
            }
            const unsigned m = __ballot_sync(full, starts);
            if (starts) st->seg[side][ns + __popc(m & ((1u << lane) - 1u))] = (uint8_t)k;
            ns += __popc(m);
        }
        if (lane == 0) st->nseg[side] = ns;
        __syncwarp();
        *at += n;
        if (*at >= total) {
            *g += 32;
            *at = 0;
        } else {
            *at -= 1;
        }
        return n;
    }
    return 0;
}

// Staged segments of side gs against the np staged points of the other: a
// segment per lane, a group of R < 32 of them repeated over floor(32 / R)
// slices of lanes that share the points.
template <bool kGeo>
__device__ bool staged_near(const WStage *st, int gs, uint32_t np, const Near &w, int lane, uint32_t &tests,
                            uint32_t &rechk) {
    const unsigned full = 0xffffffffu;
    const float4 *pt = st->pt[gs ^ 1];
    const uint32_t ns = st->nseg[gs];
    for (uint32_t k0 = 0; k0 < ns; k0 += 32) {
        const uint32_t R = min(32u, ns - k0);
        const uint32_t G = 32u / R, slice = (uint32_t)lane / R;
        const bool valid = slice < G;
        Seg g{};
        if (valid) {
            const uint32_t at = st->seg[gs][k0 + (uint32_t)lane % R];
            const float4 a = st->pt[gs][at], b = st->pt[gs][at + 1];
            g = make_seg(make_float2(a.x, a.y), make_float2(b.x, b.y));
        }
        const uint32_t q = (np + G - 1) / G;
        const uint32_t j0 = valid ? min(np, slice * q) : np, j1 = min(np, j0 + q);
        tests += j1 - j0;
        bool may = false, hit = false;
#pragma unroll 1
        for (uint32_t j = j0; j < j1; j++) {
            const float4 p = pt[j];
            screen<kGeo>(make_float2(p.x, p.y), make_float2(p.z, p.w), g, w, may, hit);
        }
        if (__any_sync(full, hit)) return true;
        if (!__any_sync(full, may)) continue;
        for (uint32_t j = j0; may && j < j1 && !hit; j++) {
            const float4 p = pt[j];
            bool here = false, sure = false;
            screen<kGeo>(make_float2(p.x, p.y), make_float2(p.z, p.w), g, w, here, sure);
            if (!here) continue;
            rechk++;
            hit = pt_seg_dist(make_float2(p.x, p.y), g.p1, g.p2, kGeo) < w.thr;
        }
        if (__any_sync(full, hit)) return true;
    }
    return false;
}

// One candidate by the warp: every point of one side against every segment of
// the other, both ways.
template <bool kGeo>
__device__ __noinline__ bool warp_near(const SeqSet &A, const SeqSet &B, const Near &w, const float2 *tab, WStage *st,
                                       int lane, uint32_t &tests, uint32_t &rechk) {
    uint32_t ga = 0, ata = 0;
    for (uint32_t na; (na = stage_points<kGeo>(A, st, 0, tab, &ga, &ata, lane)) != 0;) {
        uint32_t gb = 0, atb = 0;
#pragma unroll 1
        for (uint32_t nb; (nb = stage_points<kGeo>(B, st, 1, tab, &gb, &atb, lane)) != 0;)
#pragma unroll 1
            for (int side = 0; side < 2; side++)
                if (staged_near<kGeo>(st, side, side ? na : nb, w, lane, tests, rechk)) return true;
    }
    return false;
}

struct WithinTally {
    unsigned long long cand = 0, box = 0, tests = 0, rechk = 0, seqp = 0;
};

// Candidates (one per lane, valid lanes) against the threshold, the warp on one
// at a time: the mask of lanes whose pixel pair holds a point-segment distance
// below it. (A lane per candidate, its points read one by one, took 1.1x to 1.4x
// the time: 32 lanes at 32 places wait for every load.)
__device__ __noinline__ unsigned test_candidates(const StoreView &sv, const PolyHdr &S, const PolyHdr &T, bool valid,
                                                 uint32_t id1, uint32_t id2, const Near &w, bool geo, const float2 *tab,
                                                 WStage *stage, int lane, WithinTally &my) {
    const unsigned full = 0xffffffffu;
    SeqSet A{}, B{};
    if (valid) {
        A = seq_set(sv, S, id1);
        B = seq_set(sv, T, id2);
        my.seqp += (unsigned long long)(A.b - A.a) * (B.b - B.a);
    }
    uint32_t tests = 0, rechk = 0;
    unsigned hits = 0;
#pragma unroll 1
    for (unsigned m = __ballot_sync(full, valid); m; m &= m - 1) {
        const int src = __ffs(m) - 1;
        const SeqSet a{sv.seq + S.seq, sv.ring + S.ring, __shfl_sync(full, A.a, src), __shfl_sync(full, A.b, src)};
        const SeqSet b{sv.seq + T.seq, sv.ring + T.ring, __shfl_sync(full, B.a, src), __shfl_sync(full, B.b, src)};
        const bool h = geo ? warp_near<true>(a, b, w, tab, stage, lane, tests, rechk)
                           : warp_near<false>(a, b, w, tab, stage, lane, tests, rechk);
        if (h) hits |= 1u << src;
    }
    my.tests += tests;
    my.rechk += rechk;
    return hits;
}

enum : uint8_t { W_FALSE = 0, W_TRUE = 1, W_BADPOLY = 2 };

struct WithinArgs {
    const uint32_t *pairs;
    const uint32_t *order;  // pairs taken in this order, or index order
    uint64_t n;
    uint64_t tgt_base;
    double thr;
    bool geo, approx;
    uint32_t cap_pix;  // per-side pixel capacity of a warp's scratch
    uint32_t *scratch; // per warp (within_scratch_words)
    uint64_t scratch_words;
    uint8_t *out;
    unsigned long long *next;
    unsigned long long *stats;  // candidates, box pairs, tests, FP64 tests, sequence pairs
    SpillPool sp;
};

// A layer of a polygon's hierarchy (layer_geom), the parts the descent reads.
struct Layer {
    double mbr[2], step_x, step_y;
    int32_t dimx, dimy;
    uint32_t offset, pad;
};
constexpr int kMaxLayers = 32;

// All layers of a polygon into L, a lane each: every layer's box and dims come
// from the finest raster directly (its step is the finest one doubled, which
// is exact), and its status offset is the finer layers' sizes added up.
__device__ __noinline__ void load_layers(const PolyHdr &h, Layer *L, int lane) {
    const unsigned full = 0xffffffffu;
    const int nl = (int)h.num_layers, up = nl - 1 - lane;
    Layer g{};
    uint32_t size = 0;
    if (up == 0) {
        g.mbr[0] = h.mbr[0];
        g.mbr[1] = h.mbr[1];
        g.step_x = h.step_x;
        g.step_y = h.step_y;
        g.dimx = h.dimx;
        g.dimy = h.dimy;
    } else if (up > 0) {
        g.step_x = ldexp(h.step_x, up);
        g.step_y = ldexp(h.step_y, up);
        g.mbr[0] = floor(h.mbr[0] / g.step_x) * g.step_x;
        g.mbr[1] = floor(h.mbr[1] / g.step_y) * g.step_y;
        const double hx = ceil(h.mbr[2] / g.step_x) * g.step_x, hy = ceil(h.mbr[3] / g.step_y) * g.step_y;
        g.dimx = (int)round((hx - g.mbr[0]) / g.step_x);
        g.dimy = (int)round((hy - g.mbr[1]) / g.step_y);
        size = (uint32_t)(g.dimx * g.dimy);
    }
    uint32_t incl = size;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += u;
    }
    const uint32_t all = __shfl_sync(full, incl, 31);
    if (up > 0) g.offset = h.P + (all - incl);
    if (lane < nl) L[lane] = g;
}

__device__ __forceinline__ Box layer_box(const Layer &g, int id) {
    const int x = id % g.dimx, y = id / g.dimx;
    Box b;
    b.lo0 = g.mbr[0] + x * g.step_x;
    b.lo1 = g.mbr[1] + y * g.step_y;
    b.hi0 = g.mbr[0] + (x + 1) * g.step_x;
    b.hi1 = g.mbr[1] + (y + 1) * g.step_y;
    return b;
}

struct SideScratch {
    uint32_t *bits;  // cap_pix/32 + 1 words
    uint32_t *q;     // current queued set
    uint32_t *p;     // next level set
    float4 *fbox;    // float corners (lo0, lo1, hi0, hi1) of the pixels in p
    float *lon;      // geography, source side: longitude scale at lo1
};

// u32 words of one warp's scratch: per side the float corners (4 words each)
// of up to cap pixels, the source side's scales, per side a bitmap and two lists
__host__ __device__ inline uint64_t within_scratch_words(uint32_t cap) {
    const uint64_t w = 9ull * cap + 2 * (((uint64_t)cap >> 5) + 1 + 2ull * cap);
    return (w + 3) & ~3ull;
}

__device__ __forceinline__ void set_bit(uint32_t *bits, uint32_t id) { atomicOr(&bits[id >> 5], 1u << (id & 31)); }

// Compact the set bits of [0, nbits) into list (ascending) and clear them.
__device__ __noinline__ uint32_t compact_bits(uint32_t *bits, uint32_t nbits, uint32_t *list, int lane) {
    uint32_t nw = (nbits + 31) >> 5;
    uint32_t total = 0;
#pragma unroll 1
    for (uint32_t w0 = 0; w0 < nw; w0 += 32) {
        uint32_t w = w0 + lane;
        uint32_t word = w < nw ? bits[w] : 0u;
        uint32_t c = __popc(word);
        uint32_t incl = c;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        uint32_t at = total + incl - c;
        while (word) {
            int b = __ffs(word) - 1;
            list[at++] = (w << 5) + b;
            word &= word - 1;
        }
        if (w < nw) bits[w] = 0u;
        total += __shfl_sync(0xffffffffu, incl, 31);
    }
    __syncwarp();
    return total;
}

// Children of the queued pixels at layer g (their box at the coarser layer pg,
// shrunk by 1e-6, then retrieve_pixels' own 1e-6) or the queued pixels
// themselves; BORDER ones only (Ideal.cpp:2513-2551).
__device__ __noinline__ uint32_t next_set(const PolyHdr &h, const uint8_t *status, const Layer &g, const Layer *pg, uint32_t nq,
                             SideScratch &sc, int lane, int cc) {
    const uint8_t *st = status + h.st + g.offset;
#pragma unroll 1
    for (uint32_t k = lane; k < nq; k += 32) {
        uint32_t id = sc.q[k];
        if (pg) {
            Box b = layer_box(*pg, (int)id);
            b.lo0 += 1e-6;
            b.lo1 += 1e-6;
            b.hi0 -= 1e-6;
            b.hi1 -= 1e-6;
            int sx = offset_x(g.mbr, g.step_x, g.dimx, b.lo0 + 1e-6);
            int sy = offset_y(g.mbr, g.step_y, g.dimy, b.lo1 + 1e-6);
            int ex = offset_x(g.mbr, g.step_x, g.dimx, b.hi0 - 1e-6);
            int ey = offset_y(g.mbr, g.step_y, g.dimy, b.hi1 - 1e-6);
#pragma unroll 1
            for (int x = sx; x <= ex; x++)
#pragma unroll 1
                for (int y = sy; y <= ey; y++) {
                    uint32_t c = (uint32_t)(y * g.dimx + x);
                    if (show_status(st[c], cc) == 1) set_bit(sc.bits, c);
                }
        } else if (show_status(st[id], cc) == 1) {
            set_bit(sc.bits, id);
        }
    }
    __syncwarp();
    return compact_bits(sc.bits, (uint32_t)(g.dimx * g.dimy), sc.p, lane);
}

// The pairs (k1, k2) of [0, ns) x [0, nt) in batches of 32 lanes: the longer
// list over the lanes, the other in the outer loop; two short ones are
// flattened. One loop body serves all three (k_within's code would otherwise
// not stay in the instruction cache).
struct Product {
    uint32_t ns, nt, outer, inner, o = 0, b = 0;
    int way;  // 0 flat, 1 targets over the lanes, 2 sources over the lanes
    __device__ __forceinline__ Product(uint32_t ns_, uint32_t nt_) : ns(ns_), nt(nt_) {
        way = nt >= ns && nt >= 24 ? 1 : (ns >= 24 ? 2 : 0);
        outer = way == 0 ? 1u : (way == 1 ? ns : nt);
        inner = way == 0 ? ns * nt : (way == 1 ? nt : ns);
        if (ns == 0 || nt == 0) outer = 0;
    }
    // this lane's pair of the next batch; false past the last
    __device__ __forceinline__ bool next(int lane, uint32_t &k1, uint32_t &k2, bool &valid) {
        if (o >= outer) return false;
        const uint32_t k = b + lane;
        valid = k < inner;
        k1 = way == 0 ? k / nt : (way == 1 ? o : k);
        k2 = way == 0 ? k - k1 * nt : (way == 1 ? k : o);
        b += 32;
        if (b >= inner) {
            b = 0;
            o++;
        }
        return true;
    }
};

// FP32 view of one level's box pairs. Float corners are off by half an ulp of
// the coordinate, so a box distance computed from them is off by at most
// slack(k1) plus 4e-6 of itself; max-distances use the reference's own float
// corners and are off by 4e-6 of themselves (scales and squares).
template <bool kGeo>
struct Level {
    float ex, ey;  // coordinate roundings, x and y
    const float *lon;
    __device__ __forceinline__ float sx(uint32_t k1) const { return kGeo ? lon[k1] : 1.f; }
    __device__ __forceinline__ float sy() const { return kGeo ? (float)(40076.0 / 360.0) : 1.f; }
    __device__ __forceinline__ float slack(float sx_) const { return 1.5f * (ex * sx_ + ey * sy()); }
    __device__ __forceinline__ float dist(const float4 &a, const float4 &t, float sx_) const {
        const float dx = fmaxf(0.f, fmaxf(t.x - a.z, a.x - t.z)) * sx_;
        const float dy = fmaxf(0.f, fmaxf(t.y - a.w, a.y - t.w)) * sy();
        return sqrtf(__fmaf_rn(dx, dx, dy * dy));
    }
    __device__ __forceinline__ float max2(const float4 &a, const float4 &t, float sx_) const {
        const float2 m = corner_spans(a, t);
        const float dx = m.x * sx_, dy = m.y * sy();
        return __fmaf_rn(dx, dx, dy * dy);
    }
    // below every value the distance can have
    __device__ __forceinline__ float low(float d, float sx_) const { return d * (1.f - 4e-6f) - slack(sx_); }
    __device__ __forceinline__ float high(float d, float sx_) const { return d * (1.f + 4e-6f) + slack(sx_); }
};

__device__ __forceinline__ float warp_min(float v) {
    for (int o = 16; o; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Keep the pixels of a side whose box may lie within `cut` of box bb.
template <bool kGeo>
__device__ __noinline__ uint32_t prune_side(SideScratch &sc, uint32_t n, const float4 &bb, const Level<kGeo> &lv,
                                            bool source, float sx_low, float cut, int lane) {
    uint32_t at = 0;
#pragma unroll 1
    for (uint32_t b = 0; b < n; b += 32) {
        const uint32_t k = b + lane;
        bool keep = false;
        uint32_t id = 0;
        float4 fb = make_float4(0, 0, 0, 0);
        float lo = 0;
        if (k < n) {
            id = sc.p[k];
            fb = sc.fbox[k];
            if (source && kGeo) lo = sc.lon[k];
            const float sx_ = source ? (kGeo ? lo : 1.f) : sx_low;
            keep = !(lv.low(lv.dist(fb, bb, sx_), source ? sx_ : (kGeo ? kScaleGeo : 1.f)) > cut);
        }
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
            const uint32_t w = at + __popc(m & ((1u << lane) - 1));
            sc.p[w] = id;
            sc.fbox[w] = fb;
            if (source && kGeo) sc.lon[w] = lo;
        }
        at += __popc(m);
        __syncwarp();
    }
    return at;
}

// The reference's order of candidates (Ideal.cpp:2612).
struct CandKey {
    double apx, lo, hi;
    int32_t id1, id2;
};
__device__ __forceinline__ bool key_less(const CandKey &a, const CandKey &b) {
    if (a.apx != b.apx) return a.apx < b.apx;
    if (a.lo != b.lo) return a.lo < b.lo;
    if (a.hi != b.hi) return a.hi < b.hi;
    if (a.id1 != b.id1) return a.id1 < b.id1;
    return a.id2 < b.id2;
}

// A pair's finest level, for the candidates' FP64 expressions.
struct Finest {
    const StoreView *sv;
    const PolyHdr *S, *T;
    const Layer *gs, *gt;
    bool geo;
};
__device__ __noinline__ double exact_lo(const Finest &f, uint32_t id1, uint32_t id2) {
    return box_distance(layer_box(*f.gs, (int)id1), layer_box(*f.gt, (int)id2), f.geo);
}
__device__ __noinline__ double exact_hi(const Finest &f, uint32_t id1, uint32_t id2) {
    const Box b = layer_box(*f.gs, (int)id1);
    return box_max_distance_f(box_corners_f(b), box_corners_f(layer_box(*f.gt, (int)id2)), b.lo1, f.geo);
}
__device__ __noinline__ CandKey cand_key(const Finest &f, uint32_t id1, uint32_t id2) {  // Ideal.cpp:2587-2606
    CandKey c;
    c.id1 = (int32_t)id1;
    c.id2 = (int32_t)id2;
    c.lo = exact_lo(f, id1, id2);
    c.hi = exact_hi(f, id1, id2);
    const PolyHdr &S = *f.S, &T = *f.T;
    const int pf = classify(f.sv->areas[S.pix + id1] + f.sv->areas[T.pix + id2],
                            S.step_x * S.step_y + T.step_x * T.step_y, 20);
    c.apx = c.lo + (double)c_mean20[pf] * (c.hi - c.lo);
    return c;
}

struct WithinShared {
    WStage stage[8];
    Layer layers[8][2][kMaxLayers];
    uint2 queue[8][kQueue];
    float2 tab[900];  // longitude entries, geography only
};

// The sequence pairs of candidate (id1, id2), the last in order, from the
// *from-th on (skipped ones not counted): 1 when the next one holds a distance
// below the threshold, 0 when it ends the search (its minimum is below the
// running minimum's start value, or there is none), 2 when it does neither.
// Both questions are the staged tests' of one sequence against one, so no
// product of two lengths is formed (a single-pixel polygon's sequence is its
// whole ring, and two of 46,342 vertices make 2^32 tests).
template <bool kGeo>
__device__ __noinline__ int last_pair(const Finest &f, uint32_t id1, uint32_t id2, double thr, uint32_t *from, int lane,
                                      WithinTally &my) {
    extern __shared__ __align__(16) unsigned char within_smem[];
    WithinShared &sh = *reinterpret_cast<WithinShared *>(within_smem);
    WStage *stage = &sh.stage[threadIdx.x >> 5];
    SeqSet A = seq_set(*f.sv, *f.S, id1), B = seq_set(*f.sv, *f.T, id2);
    const uint32_t b0 = B.a, b1 = B.b;
    uint32_t at = 0;
#pragma unroll 1
    for (const uint32_t a1 = A.b; A.a < a1; A.a++) {
#pragma unroll 1
        for (B.a = b0; B.a < b1; B.a++) {
            if (A.seq[A.a].y < 2 || B.seq[B.a].y < 2) continue;
            if (at++ < *from) continue;
            (*from)++;
            A.b = A.a + 1;
            B.b = B.a + 1;
            uint32_t tests = 0, rechk = 0;
            int r = 1;  // below the threshold (1), or else below the start value (0)?
#pragma unroll 1
            for (; r >= 0; r--)
                if (warp_near<kGeo>(A, B, near_of(*f.S, *f.T, r ? thr : 100000.0, kGeo), sh.tab, stage, lane, tests,
                                    rechk))
                    break;
            my.tests += tests;
            my.rechk += rechk;
            return r < 0 ? 2 : r;
        }
    }
    return 0;
}

// resident blocks of k_within per SM (its grid, and so its scratch)
constexpr int kWithinBlocks = 2;
// box pairs of a level above which its pixel sets are pruned first
constexpr uint32_t kPrunePairs = 256;

// One warp per pair.
//
// Descent: what bounds it is the FP64 pipe (2 lanes per clock per SM against
// 128 for FP32), so the box distances of a level are screened in FP32 with
// error bounds, and the reference's FP64 expressions decide only what the
// screen leaves open: the smallest max-distance among the pairs within 1e-5
// of the FP32 smallest, and the kept pairs within the rounding of the cut. A
// large level first drops pixels that lie farther from the other polygon's
// box than a max-distance already found: they can be in neither the smallest
// max-distance nor a kept pair.
//
// Refinement: the candidates' points staged in shared memory, a segment per
// lane; first the closest candidate each lane met, then all, up to the budget;
// the rest is spilled.
//
// 60,001 pairs of configuration 3: 794 ms refinement and 55 ms descent with an
// ordered refinement, a warp per pair; 29 ms in all so (36 ms with a lane per
// candidate and every hit confirmed in FP64). What was left waited for
// instruction fetch more than for anything else: short loops are not unrolled
// and each metric has a kernel of its own (223 -> 150 KB of code, 26 ms).
template <bool kGeo>
__global__ void __launch_bounds__(256, kWithinBlocks) k_within(const StoreView sv, WithinArgs a) {
    extern __shared__ __align__(16) unsigned char within_smem[];
    WithinShared &sh = *reinterpret_cast<WithinShared *>(within_smem);
    float2 *tab = sh.tab;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    WStage *stage = &sh.stage[wib];
    const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int cc = sv.category_count;
    constexpr bool geo = kGeo;
    uint2 *q = sh.queue[wib];
    Layer *LS = sh.layers[wib][0], *LT = sh.layers[wib][1];
    if (geo)
#pragma unroll 1
        for (int k = threadIdx.x; k < 900; k += blockDim.x) tab[k] = lon_entry(k);
    const uint32_t cap = a.cap_pix, bw = (cap >> 5) + 1;
    uint32_t *wbase = a.scratch + warp * a.scratch_words;
    float4 *fboxes = reinterpret_cast<float4 *>(wbase);
    uint32_t *base = wbase + 9ull * cap;
    SideScratch ss{base, base + bw, base + bw + cap, fboxes, reinterpret_cast<float *>(wbase + 8ull * cap)};
    SideScratch ts{base + bw + 2 * cap, base + 2 * bw + 2 * cap, base + 2 * bw + 3 * cap, fboxes + cap, nullptr};
#pragma unroll 1
    for (uint32_t w = lane; w < bw; w += 32) ss.bits[w] = ts.bits[w] = 0u;
    __syncthreads();
    WithinTally my;
    for (;;) {
        unsigned long long pid = 0;
        if (lane == 0) {
            pid = atomicAdd(a.next, 1ull);
            if (a.order && pid < a.n) pid = a.order[pid];
        }
        pid = __shfl_sync(full, pid, 0);
        if (pid >= a.n) break;
        const PolyHdr &S = sv.hdr[a.pairs[2 * pid]];
        const PolyHdr &T = sv.hdr[a.tgt_base + a.pairs[2 * pid + 1]];
        if (S.err || T.err) {
            if (lane == 0) a.out[pid] = W_BADPOLY;
            continue;
        }
        __syncwarp();
        load_layers(S, LS, lane);
        load_layers(T, LT, lane);
        __syncwarp();
        const uint32_t sL = S.num_layers - 1, tL = T.num_layers - 1;
        // initial queue: every layer-0 pixel pair (Ideal.cpp:2483-2488)
        uint32_t nqs = (uint32_t)(LS[0].dimx * LS[0].dimy), nqt = (uint32_t)(LT[0].dimx * LT[0].dimy);
#pragma unroll 1
        for (uint32_t k = lane; k < nqs; k += 32) ss.q[k] = k;
#pragma unroll 1
        for (uint32_t k = lane; k < nqt; k += 32) ts.q[k] = k;
        __syncwarp();
        uint32_t i = 0, j = 0;
        bool yes = false, spilled = false;
        uint32_t head = 0;
        for (;;) {
            const double s_step = LS[i].step_x, t_step = LT[j].step_x;
            bool s_next = false, t_next = false;
            if (i < sL && (s_step >= t_step || j >= tL)) {
                i++;
                s_next = true;
            }
            if (j < tL && (s_step <= t_step || i >= sL)) {
                j++;
                t_next = true;
            }
            if (nqs == 0 || nqt == 0) break;  // empty queue
            const Layer &gs = LS[i], &gt = LT[j];
            uint32_t ns = next_set(S, sv.status, gs, s_next ? &LS[i - 1] : nullptr, nqs, ss, lane, cc);
            uint32_t nt = next_set(T, sv.status, gt, t_next ? &LT[j - 1] : nullptr, nqt, ts, lane, cc);
            if (ns == 0 || nt == 0) break;
            if (lane == 0) my.box += (uint64_t)ns * nt;
#pragma unroll 1
            for (uint32_t k = lane; k < ns; k += 32) {
                const Box b = layer_box(gs, (int)ss.p[k]);
                ss.fbox[k] = box_corners_f(b);
                if (geo) {
                    double l = fabs(b.lo1);
                    if (l == 90) l = 89.9;
                    const int idx = (int)(l * 10);
                    ss.lon[k] = c_inv_deg_lon_f[idx < 0 || idx >= 900 ? 899 : idx];
                }
            }
#pragma unroll 1
            for (uint32_t k = lane; k < nt; k += 32) ts.fbox[k] = box_corners_f(layer_box(gt, (int)ts.p[k]));
            __syncwarp();
            const float4 sbb = make_float4((float)gs.mbr[0], (float)gs.mbr[1], (float)(gs.mbr[0] + gs.dimx * gs.step_x),
                                           (float)(gs.mbr[1] + gs.dimy * gs.step_y));
            const float4 tbb = make_float4((float)gt.mbr[0], (float)gt.mbr[1], (float)(gt.mbr[0] + gt.dimx * gt.step_x),
                                           (float)(gt.mbr[1] + gt.dimy * gt.step_y));
            Level<kGeo> lv;
            lv.ex = 2.4e-7f * (fmaxf(fabsf(sbb.x), fabsf(sbb.z)) + fmaxf(fabsf(tbb.x), fabsf(tbb.z)));
            lv.ey = 2.4e-7f * (fmaxf(fabsf(sbb.y), fabsf(sbb.w)) + fmaxf(fabsf(tbb.y), fabsf(tbb.w)));
            lv.lon = ss.lon;
            float sx_low = 1.f;  // the smallest longitude scale of the source pixels
            if (geo) {
                sx_low = INFINITY;
#pragma unroll 1
                for (uint32_t k = lane; k < ns; k += 32) sx_low = fminf(sx_low, ss.lon[k]);
                sx_low = warp_min(sx_low);
            }
            const bool large = (uint64_t)ns * nt > kPrunePairs;
            if (large) {
                // the source pixel nearest T's box and the target pixel nearest
                // S's: the smallest max-distance of either is a first cut
                float best = INFINITY;
                uint32_t bk = 0;
#pragma unroll 1
                for (uint32_t k = lane; k < ns; k += 32) {
                    const float d = lv.dist(ss.fbox[k], tbb, lv.sx(k));
                    if (d < best) best = d, bk = k;
                }
                float w = warp_min(best);
                bk = __shfl_sync(full, bk, __ffs(__ballot_sync(full, best == w)) - 1);
                const float4 near_s = ss.fbox[bk];
                const float near_sx = lv.sx(bk);
                best = INFINITY;
                bk = 0;
#pragma unroll 1
                for (uint32_t k = lane; k < nt; k += 32) {
                    const float d = lv.dist(ts.fbox[k], sbb, sx_low);
                    if (d < best) best = d, bk = k;
                }
                w = warp_min(best);
                bk = __shfl_sync(full, bk, __ffs(__ballot_sync(full, best == w)) - 1);
                const float4 near_t = ts.fbox[bk];
                float ub2 = INFINITY;
#pragma unroll 1
                for (uint32_t k = lane; k < nt; k += 32) ub2 = fminf(ub2, lv.max2(near_s, ts.fbox[k], near_sx));
#pragma unroll 1
                for (uint32_t k = lane; k < ns; k += 32) ub2 = fminf(ub2, lv.max2(ss.fbox[k], near_t, lv.sx(k)));
                const float cut = sqrtf(warp_min(ub2)) * 1.00001f;
                ns = prune_side(ss, ns, tbb, lv, true, sx_low, cut, lane);
                nt = prune_side(ts, nt, sbb, lv, false, sx_low, cut, lane);
            }
            // smallest box max-distance; any <= d decides (Ideal.cpp:2557-2570)
            uint32_t k1, k2;
            bool v;
            float m2 = INFINITY;
            for (Product p(ns, nt); p.next(lane, k1, k2, v);)
                if (v) m2 = fminf(m2, lv.max2(ss.fbox[k1], ts.fbox[k2], lv.sx(k1)));
            m2 = warp_min(m2);
            if (sqrtf(m2) * 1.00001f < (float)a.thr * 0.999999f) {
                yes = true;
                break;
            }
            const Finest fin{&sv, &S, &T, &gs, &gt, geo};
            const float m2_lim = m2 * 1.00002f;
            double mbd = INFINITY;
            for (Product p(ns, nt); p.next(lane, k1, k2, v);)
                if (v && !(lv.max2(ss.fbox[k1], ts.fbox[k2], lv.sx(k1)) > m2_lim)) {
                    my.rechk++;
                    const double md = exact_hi(fin, ss.p[k1], ts.p[k2]);
                    mbd = md < mbd ? md : mbd;
                }
            for (int o = 16; o; o >>= 1) {
                const double u = __shfl_xor_sync(full, mbd, o);
                mbd = mbd < u ? mbd : u;
            }
            if (mbd <= a.thr) {
                yes = true;
                break;
            }
            mbd = mbd < 100000.0 ? mbd : 100000.0;  // the reference's start value
            // keep pairs with box distance <= d and < the smallest max-distance
            const float lim = (float)(a.thr < mbd ? a.thr : mbd);
            const float lim_up = lim * 1.000001f, lim_dn = lim * 0.999999f;
            if (large && (uint64_t)ns * nt > kPrunePairs) {
                ns = prune_side(ss, ns, tbb, lv, true, sx_low, lim_up, lane);
                nt = prune_side(ts, nt, sbb, lv, false, sx_low, lim_up, lane);
            }
            auto keep_pair = [&](uint32_t k1, uint32_t k2, float &d) {
                const float sx_ = lv.sx(k1);
                d = lv.dist(ss.fbox[k1], ts.fbox[k2], sx_);
                if (lv.low(d, sx_) > lim_up) return false;
                if (lv.high(d, sx_) < lim_dn) return true;
                my.rechk++;
                const double lo = exact_lo(fin, ss.p[k1], ts.p[k2]);
                return !(lo > a.thr) && lo < mbd;
            };
            float d;
            if (s_next || t_next) {
                for (Product p(ns, nt); p.next(lane, k1, k2, v);)
                    if (v && keep_pair(k1, k2, d)) {
                        set_bit(ss.bits, ss.p[k1]);
                        set_bit(ts.bits, ts.p[k2]);
                    }
                __syncwarp();
                nqs = compact_bits(ss.bits, (uint32_t)(gs.dimx * gs.dimy), ss.q, lane);
                nqt = compact_bits(ts.bits, (uint32_t)(gt.dimx * gt.dimy), ts.q, lane);
                continue;
            }
            // ---- the finest level: its kept pairs are the candidates. First
            // they are counted, and each lane keeps the closest one it meets.
            uint32_t cnt = 0, b1 = 0, b2 = 0;
            float bestd = INFINITY;
            bool apx_hit = false;
            for (Product p(ns, nt); p.next(lane, k1, k2, v);)
                if (v && keep_pair(k1, k2, d)) {
                    cnt++;
                    if (a.approx) {
                        // Within "-a" (query_within_polygon.cu:332-375): a pair left
                        // undecided is within when one of its surviving finest pixel
                        // pairs has apxDist = minDist + mean (maxDist - minDist) <=
                        // the distance, in float. mean is (1.0 - pf /
                        // category_count) * 0.5 with both operands 8-bit integers
                        // (:352), so the quotient is 0 and mean is 0.5; 0.5 (max -
                        // min) is exact in float, so contracting the sum into an FMA
                        // rounds the same.
                        const float lo = (float)exact_lo(fin, ss.p[k1], ts.p[k2]);
                        const float hi = (float)exact_hi(fin, ss.p[k1], ts.p[k2]);
                        apx_hit |= (double)(lo + 0.5f * (hi - lo)) <= a.thr;
                    } else {
                        d += sqrtf(lv.max2(ss.fbox[k1], ts.fbox[k2], lv.sx(k1)));
                        if (d < bestd) bestd = d, b1 = ss.p[k1], b2 = ts.p[k2];
                    }
                }
            my.cand += cnt;
            for (int o = 16; o; o >>= 1) cnt += __shfl_xor_sync(full, cnt, o);
            if (a.approx) {
                yes = __any_sync(full, apx_hit);
                break;
            }
            if (cnt == 0) break;
            const Near w = near_of(S, T, a.thr, geo);
            // queue of candidates (pixel ids): the closest ones, then all
            const unsigned pm = __ballot_sync(full, bestd < INFINITY);
            if (bestd < INFINITY) q[__popc(pm & ((1u << lane) - 1))] = make_uint2(b1, b2);
            int qn = __popc(pm);
            // the last candidate in order, once known: only its first sequence
            // pair counts, and it is left out of everything else
            bool know_last = false, may_spill = a.sp.cap > 0, more = cnt > (uint32_t)qn;
            uint32_t last1 = ~0u, last2 = ~0u, spent = 0;
            Product all(ns, nt);
            __syncwarp();
            for (;;) {
#pragma unroll 1
                for (int k = 0; k < qn && !yes;) {
                    bool check_last = false;
                    if (may_spill && (float)spent >= a.sp.budget) {
                        if (know_last) {
#pragma unroll 1
                            for (int e = k + lane; e < qn; e += 32)
                                if (q[e].x == last1 && q[e].y == last2) q[e].x = ~0u;
                            __syncwarp();
                            if (spill_rest(a.sp, pid, q, k, qn, 0.f, lane, &head, &spilled)) break;
                            may_spill = false;  // the pool is full
                            continue;
                        }
                        CandKey top{-1.0, 0, 0, 0, 0};  // the largest key of all
                        for (Product p(ns, nt); p.next(lane, k1, k2, v);)
                            if (v && keep_pair(k1, k2, d)) {
                                const CandKey c = cand_key(fin, ss.p[k1], ts.p[k2]);
                                if (key_less(top, c)) top = c;
                            }
                        for (int o = 16; o; o >>= 1) {
                            CandKey c;
                            c.apx = __shfl_xor_sync(full, top.apx, o);
                            c.lo = __shfl_xor_sync(full, top.lo, o);
                            c.hi = __shfl_xor_sync(full, top.hi, o);
                            c.id1 = __shfl_xor_sync(full, top.id1, o);
                            c.id2 = __shfl_xor_sync(full, top.id2, o);
                            if (key_less(top, c)) top = c;
                        }
                        last1 = (uint32_t)top.id1;
                        last2 = (uint32_t)top.id2;
                        check_last = true;
                    } else {
                        const uint2 c = k + lane < qn ? q[k + lane] : make_uint2(~0u, ~0u);
                        const bool ok = c.x != ~0u && !(know_last && c.x == last1 && c.y == last2);
                        const unsigned hits = test_candidates(sv, S, T, ok, c.x, c.y, w, geo, tab, stage, lane, my);
                        k += 32;
                        spent += 32;
                        if (hits == 0) continue;
                        yes = know_last || (hits & (hits - 1)) != 0;
                        if (yes) break;
                        // one hit: it counts unless its candidate is the last in order
                        const int src = __ffs(hits) - 1;
                        const uint32_t h1 = __shfl_sync(full, c.x, src), h2 = __shfl_sync(full, c.y, src);
                        const CandKey key = cand_key(fin, h1, h2);
                        for (Product p(ns, nt); !yes && p.next(lane, k1, k2, v);)
                            yes = __any_sync(full, v && keep_pair(k1, k2, d) &&
                                                       key_less(key, cand_key(fin, ss.p[k1], ts.p[k2])));
                        if (yes) break;
                        last1 = h1;
                        last2 = h2;
                        check_last = true;
                    }
                    if (check_last) {
                        know_last = true;
                        uint32_t from = 0;
                        int r;
#pragma unroll 1
                        while ((r = last_pair<kGeo>(fin, last1, last2, w.thr, &from, lane, my)) == 2) {
                            // the running minimum still at its start value unless
                            // an earlier candidate holds a distance below it
                            const Near far = near_of(S, T, 100000.0, geo);
                            unsigned below = 0;
                            for (Product p(ns, nt); !below && p.next(lane, k1, k2, v);) {
                                const bool ok = v && keep_pair(k1, k2, d) && !(ss.p[k1] == last1 && ts.p[k2] == last2);
                                below = test_candidates(sv, S, T, ok, ok ? ss.p[k1] : 0, ok ? ts.p[k2] : 0, far, geo,
                                                        tab, stage, lane, my);
                            }
                            if (below) break;
                        }
                        yes = r == 1;
                    }
                }
                if (yes || !more) break;
                __syncwarp();
                qn = 0;
                while (qn + 32 <= kQueue) {
                    more = all.next(lane, k1, k2, v);
                    if (!more) break;
                    const bool keep = v && keep_pair(k1, k2, d);
                    const unsigned m = __ballot_sync(full, keep);
                    if (keep) q[qn + __popc(m & ((1u << lane) - 1))] = make_uint2(ss.p[k1], ts.p[k2]);
                    qn += __popc(m);
                }
                __syncwarp();
            }
            break;
        }
        // leave the scratch bitmaps clean for the next pair
        __syncwarp();
#pragma unroll 1
        for (uint32_t w = lane; w < bw; w += 32) {
            ss.bits[w] = 0u;
            ts.bits[w] = 0u;
        }
        __syncwarp();
        if (lane == 0) {
            a.out[pid] = yes ? W_TRUE : W_FALSE;
            if (spilled && yes) a.sp.flag[head] = 1u;  // found after the spill
        }
    }
    for (int o = 16; o; o >>= 1) {
        my.cand += __shfl_xor_sync(full, my.cand, o);
        my.tests += __shfl_xor_sync(full, my.tests, o);
        my.rechk += __shfl_xor_sync(full, my.rechk, o);
        my.seqp += __shfl_xor_sync(full, my.seqp, o);
    }
    if (lane == 0) {
        atomicAdd(&a.stats[0], my.cand);
        atomicAdd(&a.stats[1], my.box);
        atomicAdd(&a.stats[2], my.tests);
        atomicAdd(&a.stats[3], my.rechk);
        atomicAdd(&a.stats[4], my.seqp);
    }
}

// The candidates that k_within spilled, a warp's worth of one chunk at a time,
// slice by slice across the chunks (as spill_units, a lane per entry).
__global__ void __launch_bounds__(256, 3) k_within_spill(const StoreView sv, WithinArgs a) {
    __shared__ float2 tab[900];
    __shared__ WStage stages[8];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    WStage *stage = &stages[threadIdx.x >> 5];
    const unsigned long long n = min(a.sp.ctr[0], (unsigned long long)a.sp.cap);
    if (n == 0) return;
    if (a.geo)
#pragma unroll 1
        for (int k = threadIdx.x; k < 900; k += blockDim.x) tab[k] = lon_entry(k);
    __syncthreads();
    const unsigned long long total = n * ((a.sp.ctr[2] + 31) / 32);
    WithinTally my;
    for (;;) {
        unsigned long long u = 0;
        if (lane == 0) u = atomicAdd(&a.sp.ctr[1], 1ull);
        u = __shfl_sync(full, u, 0);
        if (u >= total) break;
        const uint64_t c = u % n;
        const SpillChunk h = a.sp.chunk[c];
        const uint32_t e = (uint32_t)(u / n) * 32;
        if (e >= h.count) continue;
        if (__shfl_sync(full, *(volatile uint32_t *)&a.sp.flag[h.head], 0)) continue;
        const PolyHdr &S = sv.hdr[a.pairs[2 * h.pid]];
        const PolyHdr &T = sv.hdr[a.tgt_base + a.pairs[2 * h.pid + 1]];
        const uint2 cd = e + lane < h.count ? a.sp.items[c * kQueue + e + lane] : make_uint2(~0u, 0u);
        const bool v = cd.x != ~0u;
        if (test_candidates(sv, S, T, v, cd.x, cd.y, near_of(S, T, a.thr, a.geo), a.geo, tab, stage, lane, my) && lane == 0) {
            a.sp.flag[h.head] = 1u;
            a.out[h.pid] = W_TRUE;
        }
    }
    for (int o = 16; o; o >>= 1) {
        my.tests += __shfl_xor_sync(full, my.tests, o);
        my.rechk += __shfl_xor_sync(full, my.rechk, o);
        my.seqp += __shfl_xor_sync(full, my.seqp, o);
    }
    if (lane == 0) {
        atomicAdd(&a.stats[2], my.tests);
        atomicAdd(&a.stats[3], my.rechk);
        atomicAdd(&a.stats[4], my.seqp);
    }
}

// The largest layer of any polygon, in pixels: a warp per polygon, a lane per layer.
__global__ void k_within_cap(const PolyHdr *__restrict__ hdr, uint32_t npoly, unsigned long long *__restrict__ most) {
    const int lane = threadIdx.x & 31;
    unsigned long long mine = 0;
#pragma unroll 1
    for (uint32_t p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; p < npoly; p += (gridDim.x * blockDim.x) >> 5) {
        const PolyHdr &h = hdr[p];
        if (h.err || lane >= (int)h.num_layers) continue;
        LayerGeom g;
        layer_geom(h, (uint32_t)lane, g);
        mine = max(mine, (unsigned long long)(uint32_t)(g.dimx * g.dimy));
    }
    for (int o = 16; o; o >>= 1) mine = max(mine, __shfl_xor_sync(0xffffffffu, mine, o));
    if (lane == 0 && mine) atomicMax(most, mine);
}

__global__ void k_within_count(const uint8_t *__restrict__ out, uint64_t n, unsigned long long *found) {
    unsigned long long f = 0;
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (uint64_t)gridDim.x * blockDim.x)
        f += out[k] == W_TRUE;
    for (int o = 16; o; o >>= 1) f += __shfl_xor_sync(0xffffffffu, f, o);
    if ((threadIdx.x & 31) == 0 && f) atomicAdd(found, f);
}

static unsigned gbw(uint64_t n) {
    uint64_t g = (n + 255) / 256;
    uint64_t cap = 32ull * sm_count();
    if (g > cap) g = cap;
    return (unsigned)(g ? g : 1);
}

int within(farm_store *s, const uint32_t *pairs, uint64_t n, double distance, int geography, int self, int mode,
           int mem, uint8_t *out, uint64_t *found, farm_stats *st) {
    if (mode != FARM_MODE_EXACT && mode != FARM_MODE_APPROX) {
        set_error("farm_within: mode must be FARM_MODE_EXACT or FARM_MODE_APPROX");
        return FARM_EINVAL;
    }
    if (!s->rasterized || !s->ropts.hierarchy) {
        set_error("farm_within: rasterize with hierarchy first");
        return FARM_EINVAL;
    }
    if (!self && s->n_side[1] == 0) {
        set_error("farm_within: no target side loaded (or pass target_is_source)");
        return FARM_EINVAL;
    }
    FARM_TRY(check_pairs(s, pairs, n, mem, self != 0, "farm_within"));
    FARM_TRY(ensure_tables(s->device));
    cudaStream_t stream = s->stream;
    const uint64_t tgt_base = self ? 0 : s->n_side[0];
    const uint32_t *dpairs = pairs;
    if (mem == FARM_MEM_HOST && n) {
        FARM_TRY(s->d_pairs.ensure(8 * n));
        FARM_CUDA(cudaMemcpyAsync(s->d_pairs.p, pairs, 8 * n, cudaMemcpyHostToDevice, stream));
        dpairs = s->d_pairs.as<uint32_t>();
    }
    uint8_t *dout = out;
    if (mem == FARM_MEM_HOST || !out) {
        FARM_TRY(s->d_out.ensure(n + 64));
        dout = s->d_out.as<uint8_t>();
    }
    FARM_TRY(s->d_counters.ensure(256));
    unsigned long long *ctr = s->d_counters.as<unsigned long long>();
    FARM_CUDA(cudaMemsetAsync(ctr, 0, 128, stream));
    int launches = 0;
    // the largest layer of any polygon bounds a warp's pixel sets
    uint32_t cap = 64;
    {
        k_within_cap<<<gbw(32ull * s->n_poly), 256, 0, stream>>>(s->d_hdr.as<PolyHdr>(), (uint32_t)s->n_poly, ctr + 15);
        FARM_CUDA(cudaGetLastError());
        launches++;
        unsigned long long most = 0;
        FARM_CUDA(cudaMemcpyAsync(&most, ctr + 15, 8, cudaMemcpyDeviceToHost, stream));
        FARM_CUDA(cudaStreamSynchronize(stream));
        if (most > cap) cap = (uint32_t)most;
        cap = (cap + 31) & ~31u;
    }
    FARM_CUDA(cudaEventRecord(s->ev[6], stream));
    if (n) {
        const uint64_t words = within_scratch_words(cap);
        uint64_t blocks = (uint64_t)sm_count() * kWithinBlocks;
        if (blocks > n) blocks = n;
        size_t freeb = 0, totb = 0;
        cudaMemGetInfo(&freeb, &totb);
        while (blocks > 8 && 4ull * words * 8 * blocks > freeb / 4) blocks /= 2;
        DevBuf &scr = s->s[Q_SCR0];
        FARM_TRY(scr.ensure(4 * words * 8 * blocks + 64));
        WithinArgs wa;
        wa.pairs = dpairs;
        wa.n = n;
        FARM_TRY(pair_order(s, dpairs, n, tgt_base, &wa.order));
        wa.tgt_base = tgt_base;
        wa.thr = distance;
        wa.geo = geography != 0;
        wa.approx = mode == FARM_MODE_APPROX;
        wa.cap_pix = cap;
        wa.scratch = scr.as<uint32_t>();
        wa.scratch_words = words;
        wa.out = dout;
        wa.next = ctr;
        wa.stats = ctr + 1;
        FARM_TRY(spill_pool(s, n, ctr + 8, 64.f, 512.f, &wa.sp));
        const auto kernel = wa.geo ? k_within<true> : k_within<false>;
        FARM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WithinShared)));
        kernel<<<(unsigned)blocks, 256, sizeof(WithinShared), stream>>>(s->view(), wa);
        FARM_CUDA(cudaGetLastError());
        FARM_CUDA(cudaEventRecord(s->ev[8], stream));
        k_within_spill<<<3 * sm_count(), 256, 0, stream>>>(s->view(), wa);
        FARM_CUDA(cudaGetLastError());
        launches += 2;
    }
    FARM_CUDA(cudaEventRecord(s->ev[7], stream));
    k_within_count<<<gbw(n), 256, 0, stream>>>(dout, n, ctr + 14);
    launches++;
    unsigned long long h[16];
    FARM_CUDA(cudaMemcpyAsync(h, ctr, sizeof h, cudaMemcpyDeviceToHost, stream));
    if (mem == FARM_MEM_HOST && out && n) FARM_CUDA(cudaMemcpyAsync(out, dout, n, cudaMemcpyDeviceToHost, stream));
    FARM_CUDA(cudaStreamSynchronize(stream));
    s->launches += (uint64_t)launches;
    if (found) *found = h[14];
    if (st) {
        memset(st, 0, sizeof *st);
        st->pairs = n;
        st->found = h[14];
        st->in_hits = h[1];  // candidate pixel pairs
        st->border_pairs = h[2];
        st->segment_tests = h[3];
        st->fp64_rechecks = h[4];
        st->sequence_pairs = h[5];
        float ms = 0, ms1 = 0;
        cudaEventElapsedTime(&ms, s->ev[6], s->ev[7]);
        if (n) cudaEventElapsedTime(&ms1, s->ev[6], s->ev[8]);
        st->ms_total = ms;
        st->ms_stage[1] = ms1;       // the descent and the tests kept with it
        st->ms_stage[2] = ms - ms1;  // the spilled tests
        st->kernel_launches = launches;
    }
    return FARM_OK;
}

}  // namespace farm

extern "C" int farm_within(farm_store *s, const uint32_t *pairs, uint64_t n, double distance, int geography,
                           int target_is_source, int mem, uint8_t *out, uint64_t *found, farm_stats *st) {
    using namespace farm;
    if (!s || (n && !pairs)) {
        set_error("invalid arguments to farm_within");
        return FARM_EINVAL;
    }
    return within(s, pairs, n, distance, geography, target_is_source, FARM_MODE_EXACT, mem, out, found, st);
}

extern "C" int farm_within_mode(farm_store *s, const uint32_t *pairs, uint64_t n, double distance, int geography,
                                int target_is_source, int mode, int mem, uint8_t *out, uint64_t *found,
                                farm_stats *st) {
    using namespace farm;
    if (!s || (n && !pairs)) {
        set_error("invalid arguments to farm_within_mode");
        return FARM_EINVAL;
    }
    return within(s, pairs, n, distance, geography, target_is_source, mode, mem, out, found, st);
}
