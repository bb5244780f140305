// Segment predicates and the warp-cooperative pixel-pair refinement shared
// by the intersect and contain queries.
//
//   segment_intersect (geometry_computation.h:215-221) with Point::cross
//   (Point.h:93-97) in FP32 without fused multiply-add, inter1
//   (geometry_computation.h:195-212), retrieve_pixels (MyRaster.cpp:332-346)
//   and segment_intersect_batch over two pixels' edge sequences
//   (geometry_computation.h:224-237).
#pragma once

#include "common.cuh"

namespace farm {

// Point.h:93-97: (a - o) x (b - o) in float, no fused multiply-add
__device__ __forceinline__ float cross3(float2 o, float2 a, float2 b) {
    float ax = __fsub_rn(a.x, o.x), ay = __fsub_rn(a.y, o.y);
    float bx = __fsub_rn(b.x, o.x), by = __fsub_rn(b.y, o.y);
    return __fsub_rn(__fmul_rn(ax, by), __fmul_rn(ay, bx));
}

__device__ __forceinline__ int sgnf(float x) { return x >= 0 ? (x != 0 ? 1 : 0) : -1; }

__device__ __forceinline__ bool inter1(double a, double b, double c, double d) {
    double t;
    if (a > b) { t = a; a = b; b = t; }
    if (c > d) { t = c; c = d; d = t; }
    return fmax(a, c) <= fmin(b, d);
}

// geometry_computation.h:215-221
__device__ __forceinline__ bool seg_intersect(float2 a, float2 b, float2 c, float2 d) {
    if (cross3(c, a, d) == 0.0f && cross3(c, b, d) == 0.0f)
        return inter1(a.x, b.x, c.x, d.x) && inter1(a.y, b.y, c.y, d.y);
    return sgnf(cross3(a, b, c)) != sgnf(cross3(a, b, d)) && sgnf(cross3(c, d, a)) != sgnf(cross3(c, d, b));
}

struct Window {
    int sx, ex, sy, ey;
};

// MyRaster.cpp:332-346
__device__ __forceinline__ Window retrieve(const double *mbr, double stx, double sty, int dimx, int dimy,
                                           double b0, double b1, double b2, double b3) {
    Window w;
    w.sx = offset_x(mbr, stx, dimx, b0 + 1e-6);
    w.sy = offset_y(mbr, sty, dimy, b1 + 1e-6);
    w.ex = offset_x(mbr, stx, dimx, b2 - 1e-6);
    w.ey = offset_y(mbr, sty, dimy, b3 - 1e-6);
    return w;
}

__device__ __forceinline__ int sgn_code(float v) { return (v > 0.f) - (v < 0.f); }

// (b - o) x (p - o) with e = b - o precomputed: the same roundings as cross3(o, b, p)
__device__ __forceinline__ float cross_e(float2 o, float ex, float ey, float2 p) {
    return __fsub_rn(__fmul_rn(ex, __fsub_rn(p.y, o.y)), __fmul_rn(ey, __fsub_rn(p.x, o.x)));
}

__device__ __forceinline__ bool inter1f(float a, float b, float c, float d) {
    return fmaxf(fminf(a, b), fminf(c, d)) <= fminf(fmaxf(a, b), fmaxf(c, d));
}

// exclusive warp scan of cnt; total of all lanes in `total`
__device__ __forceinline__ uint32_t warp_excl_scan(uint32_t cnt, int lane, uint32_t &total) {
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    total = __shfl_sync(0xffffffffu, incl, 31);
    return incl - cnt;
}

// the last lane whose exclusive prefix is <= item (the lane that owns item)
__device__ __forceinline__ int warp_owner(uint32_t excl, uint32_t item) {
    int owner = 0;
#pragma unroll
    for (int b = 16; b; b >>= 1) {
        int cand = owner + b;
        uint32_t ex = __shfl_sync(0xffffffffu, excl, cand);
        if (ex <= item) owner = cand;
    }
    return owner;
}

// ---------------------------------------------------- packed float pairs --
// Two floats in one 64-bit register pair: the packed FP32 instructions round
// each half as the scalar ones do, at one issue slot for both.
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t f2_sub(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Target vertices staged per warp: vertex j as (x, x, y, y) at tbuf[2j] and
// its difference from the vertex before it as (dx, dx, dy, dy) at
// tbuf[2j + 1], the broadcast operands of the packed instructions. A vertex
// that ends no segment (a sequence's first) carries kNoSegment as difference.
constexpr uint32_t kStage = 64;
constexpr uint32_t kNoSegment = 0x7fc0beefu;  // a NaN no subtraction produces
// Coordinates past this magnitude (or not finite) take the scalar walk.
constexpr float kBigCoord = 1e15f;
__device__ __forceinline__ bool big_coord(float2 p) {
    return !(fabsf(p.x) < kBigCoord && fabsf(p.y) < kBigCoord);
}

// segment_intersect of a -> b with the staged segments ending at vertices
// [jb, j1) by the reference's sign codes and its collinear interval test
// (inter1, geometry_computation.h:195-212): the walk for the rare stages in
// which a cross product is exactly zero.
static __device__ __noinline__ bool walk_signs(float2 a, float2 b, const float4 *tbuf, uint32_t jb, uint32_t j1) {
    const float ex = __fsub_rn(b.x, a.x), ey = __fsub_rn(b.y, a.y);
    bool hit = false;
    for (uint32_t j = jb; j < j1; j++) {
        const float4 e = tbuf[2 * j + 1];
        if (__float_as_uint(e.x) == kNoSegment) continue;
        const float4 c4 = tbuf[2 * j - 2], d4 = tbuf[2 * j];
        const float2 c = make_float2(c4.x, c4.z), d = make_float2(d4.x, d4.z);
        const float ux = __fsub_rn(c.x, a.x), uy = __fsub_rn(c.y, a.y);
        const float wx = __fsub_rn(c.x, b.x), wy = __fsub_rn(c.y, b.y);
        const int sya = sgn_code(__fsub_rn(__fmul_rn(e.x, uy), __fmul_rn(e.z, ux)));
        const int syb = sgn_code(__fsub_rn(__fmul_rn(e.x, wy), __fmul_rn(e.z, wx)));
        if ((sya | syb) == 0) {
            hit |= inter1f(a.x, b.x, c.x, d.x) && inter1f(a.y, b.y, c.y, d.y);
        } else if (sya != syb) {
            const int sxc = sgn_code(__fsub_rn(__fmul_rn(ex, uy), __fmul_rn(ey, ux)));
            const int sxd = sgn_code(cross_e(a, ex, ey, d));
            hit |= sxc != sxd;
        }
    }
    return hit;
}

// Refine one BORDER x BORDER pixel pair: true iff some segment of the source
// pixel's edge sequences intersects some segment of the target pixel's
// (segment_intersect_batch over every sequence pair, geometry_computation.h:
// 215-237; the reference stops at the first hit, so the set of segment pairs
// it tests differs only in where it stops, and the boolean is the same).
//
// The warp stages up to kStage target vertices in shared memory, then takes
// the source pixel's segments 32 at a time, a segment (a, b) per lane, and
// walks the staged vertices, which every lane reads as broadcasts.
// segment_intersect's four cross products are shared along the walk without
// changing a single rounding:
//   a.cross(b, c) is computed once per target vertex c and reused for the two
//     target segments that end at c;
//   c.cross(a, d) = -(c.cross(d, a)) exactly (the two products are the same
//     IEEE products and round-to-nearest is symmetric), so the collinear test
//     c.cross(a,d) == 0 && c.cross(b,d) == 0 reads the signs of c.cross(d, a)
//     and c.cross(d, b) that the general test needs anyway;
//   for the target segment c -> d, c.cross(d, a) = (d-c) x (a-c) takes the
//     differences a - c, which are the exact negations of the differences
//     c - a the lane formed one vertex earlier for a.cross(b, c);
//   the target segment's own d - c is formed once, by the lane that stages d.
// What bounds it is instruction issue, so the walk is written for few
// instructions a test: the a side and the b side ride in one packed
// instruction (5 packed and 3 scalar float instructions instead of 13), and
// signs are compared by their bits, ((s_c ^ s_d) & (p_a ^ p_b)) < 0 for a
// crossing, with one running minimum of the magnitudes. Sign bits are the
// reference's sign codes unless a value is exactly 0; then the minimum is 0
// and the lanes walk the stage again by sign codes (walk_signs). A difference
// of kNoSegment makes both products the same NaN: never a crossing, and
// ignored by the minimum.
//
// A group of R < 32 source segments (a pixel's last group, or a small pixel)
// would leave lanes idle for the whole target walk, so the group is repeated
// across G = floor(32 / R) slices of lanes and each slice walks its share of
// the staged vertices, starting from the vertex before its share. Every
// (source segment, target segment) pair is still tested once. A stage that
// ends inside a sequence is followed by one that starts with its last vertex.
//
// With nparts > 1 the call takes the source groups part, part + nparts, ...
// only, so that several warps can share one heavy pixel pair.
static __device__ bool refine_pixel_pair(const StoreView &sv, const PolyHdr &S, const PolyHdr &T, uint32_t pa,
                                         uint32_t pb, float4 *tbuf, unsigned long long &tests, uint32_t part = 0,
                                         uint32_t nparts = 1) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t *so = sv.offset + S.off, *to = sv.offset + T.off;
    const uint32_t a0 = so[pa], a1 = so[pa + 1], b0 = to[pb], b1 = to[pb + 1];
    const uint2 *sseq = sv.seq + S.seq, *tseq = sv.seq + T.seq;
    const float2 *sr = sv.ring + S.ring, *tr = sv.ring + T.ring;
    for (uint32_t tg = b0; tg < b1; tg += 32) {
        const uint32_t kk = tg + lane;
        const uint2 r2 = kk < b1 ? tseq[kk] : make_uint2(0u, 0u);
        uint32_t total2;
        const uint32_t excl2 = warp_excl_scan(kk < b1 ? r2.y + 1 : 0u, lane, total2);  // vertices
        for (uint32_t tb = 0; tb < total2; tb += kStage - 1) {
            const uint32_t m = min(kStage, total2 - tb);
            if (tb && m < 2) break;  // only the repeated vertex is left
            __syncwarp();            // the last stage's readers are done
            uint64_t segmask = 0;
            bool big = false;
            float2 last = make_float2(0.f, 0.f);
#pragma unroll
            for (uint32_t h = 0; h < kStage; h += 32) {
                const uint32_t f2 = tb + h + lane;
                const bool v2 = f2 < total2;
                const int o2 = warp_owner(excl2, f2);
                const uint32_t o_start = __shfl_sync(full, r2.x, o2), o_ex = __shfl_sync(full, excl2, o2);
                const uint32_t off = f2 - o_ex;
                float2 c = make_float2(0.f, 0.f);
                if (v2) c = tr[o_start + off];
                big |= big_coord(c);
                float px = __shfl_up_sync(full, c.x, 1), py = __shfl_up_sync(full, c.y, 1);
                if (lane == 0) {
                    px = last.x;
                    py = last.y;
                }
                const bool seg = v2 && off > 0 && h + lane > 0;  // a segment ends here
                const float none = __uint_as_float(kNoSegment);
                const float dx = seg ? __fsub_rn(c.x, px) : none, dy = seg ? __fsub_rn(c.y, py) : none;
                tbuf[2 * (h + lane)] = make_float4(c.x, c.x, c.y, c.y);
                tbuf[2 * (h + lane) + 1] = make_float4(dx, dx, dy, dy);
                segmask |= (uint64_t)__ballot_sync(full, seg) << h;
                last = make_float2(__shfl_sync(full, c.x, 31), __shfl_sync(full, c.y, 31));
                if (h + 32 >= m) break;
            }
            __syncwarp();
            uint32_t group = 0;
            for (uint32_t g = a0; g < a1; g += 32) {
                const uint32_t k = g + lane;
                const uint2 r = k < a1 ? sseq[k] : make_uint2(0u, 0u);
                uint32_t total;
                const uint32_t excl = warp_excl_scan(r.y, lane, total);  // r.y segments per sequence
                for (uint32_t sb = 0; sb < total; sb += 32, group++) {
                    if (nparts > 1 && group % nparts != part) continue;
                    // this group's R source segments, repeated over G slices of lanes
                    const uint32_t R = min(32u, total - sb);
                    const uint32_t G = 32u / R;
                    const uint32_t slice = (uint32_t)lane / R;
                    const uint32_t f = sb + (uint32_t)lane % R;
                    const bool valid = slice < G;
                    const int owner = warp_owner(excl, f);
                    const uint32_t ostart = __shfl_sync(full, r.x, owner);
                    const uint32_t oex = __shfl_sync(full, excl, owner);
                    float2 a = make_float2(0.f, 0.f), b = a;
                    if (valid) {
                        a = sr[ostart + (f - oex)];
                        b = sr[ostart + (f - oex) + 1];
                    }
                    // this slice's share [j0, j1) of the staged vertices
                    const uint32_t q = (m + G - 1) / G;
                    const uint32_t j0 = valid ? min(m, slice * q) : m, j1 = min(m, j0 + q);
                    const uint32_t jb = max(j0, 1u);  // no segment ends at the stage's first vertex
                    float z = INFINITY;
                    int acc = 0;
                    if (jb < j1) {
                        const float ex = __fsub_rn(b.x, a.x), ey = __fsub_rn(b.y, a.y);
                        const uint64_t abx = f2_pack(a.x, b.x), aby = f2_pack(a.y, b.y);
                        const ulonglong2 *tv = reinterpret_cast<const ulonglong2 *>(tbuf);
                        ulonglong2 t = tv[2 * (jb - 1)];
                        uint64_t U = f2_sub(t.x, abx), V = f2_sub(t.y, aby);
                        float ux, uy, hi;
                        f2_unpack(U, ux, hi);
                        f2_unpack(V, uy, hi);
                        float s = __fsub_rn(__fmul_rn(ex, uy), __fmul_rn(ey, ux));
                        z = fabsf(s);
#pragma unroll 4
                        for (uint32_t j = jb; j < j1; j++) {
                            t = tv[2 * j];
                            const ulonglong2 d = tv[2 * j + 1];
                            // (t - c) x (c - a) and (t - c) x (c - b), c the vertex before t
                            float pa_, pb_;
                            f2_unpack(f2_sub(f2_mul(d.x, V), f2_mul(d.y, U)), pa_, pb_);
                            U = f2_sub(t.x, abx);
                            V = f2_sub(t.y, aby);
                            f2_unpack(U, ux, hi);
                            f2_unpack(V, uy, hi);
                            const float sn = __fsub_rn(__fmul_rn(ex, uy), __fmul_rn(ey, ux));
                            acc |= (__float_as_int(s) ^ __float_as_int(sn)) &
                                   (__float_as_int(pa_) ^ __float_as_int(pb_));
                            z = fminf(fminf(z, fabsf(sn)), fminf(fabsf(pa_), fabsf(pb_)));
                            s = sn;
                        }
                        const uint64_t below = j1 >= 64 ? ~0ull : (1ull << j1) - 1ull;
                        tests += (unsigned)__popcll(segmask & below & ~((1ull << jb) - 1ull));
                    }
                    big |= big_coord(a) || big_coord(b);
                    const bool slow = __any_sync(full, z == 0.f || big);
                    if (!slow) {
                        if (__any_sync(full, acc < 0)) return true;
                    } else if (__any_sync(full, jb < j1 && walk_signs(a, b, tbuf, jb, j1))) {
                        return true;
                    }
                }
            }
        }
    }
    return false;
}

}  // namespace farm
