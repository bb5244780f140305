// Containment queries on the raster store (the reference's Ideal::contain;
// its GPU form, query_contain.cu, is commented out and never launched).
//
//   farm_contain_points: does polygon p hold point q (Ideal::contain(Point &),
//     Ideal.cpp:1101-1157). One lane per (polygon, point) pair up to its pixel,
//     the BORDER pixels' edges over all lanes of the warp: the MBR test
//     (box::contain, Box.cpp:65-70), the pixel's class, and for a BORDER pixel
//     the parity of the pixel's edges whose FP32 crossing abscissa lies in
//     [x, the pixel's right border] plus the nodes below y on the grid line at
//     that border (count_intersection_nodes, Ideal.cpp:988-1006).
//   farm_contain: does source s hold target t (Ideal::contain(Ideal *),
//     Ideal.cpp:1159-1231). One warp per candidate pair, pairs pulled from a
//     global counter: the MBR test, the source pixels' classes over t's MBR
//     window (all OUT: no; all IN: yes), then the pixel pairs under every
//     non-IN source pixel, where an OUT source pixel over an IN target pixel,
//     a target edge of a BORDER pixel crossing the border of an OUT source
//     pixel, or a crossing edge pair of BORDER x BORDER pixels means "no";
//     t's first vertex decides the rest. Every pixel-pair check can only say
//     "no", so visiting the pairs in any order gives the reference's answer.
#include <cstring>
#include <string>

#include "common.cuh"
#include "segments.cuh"
#include "spill.cuh"

namespace farm {

namespace {

constexpr int kContainWarps = 8;

struct ContainCounters {
    unsigned long long found, pixel_pairs, segment_tests;
};

// A point's pixel in polygon H (Ideal::contain(Point &); (px, py) as float, the
// reference's Point): 0 or 1 when the box or the pixel's class decides, else 2,
// with the BORDER pixel's sequences [q0, q1), the largest float up to its right
// border (a float abscissa is at most the border exactly when it is at most
// that) and the parity of the right grid line's nodes below py.
struct PointPixel {
    uint32_t q0, q1;
    float right;
    bool odd;
};
__device__ __forceinline__ int point_pixel(const StoreView &sv, const PolyHdr &H, float px, float py, PointPixel &w) {
    if (!(px >= H.mbr[0] && px <= H.mbr[2] && py >= H.mbr[1] && py <= H.mbr[3])) return 0;
    const int xo = offset_x(H.mbr, H.step_x, H.dimx, px);
    const int yo = offset_y(H.mbr, H.step_y, H.dimy, py);
    const uint32_t pix = (uint32_t)(yo * H.dimx + xo);
    const int st = show_status(sv.status[H.st + pix], sv.category_count);
    if (st == 2) return 1;
    if (st == 0) return 0;
    w.right = __double2float_rd(H.mbr[0] + (xo + 1) * H.step_x);
    const uint32_t *off = sv.offset + H.off;
    w.q0 = off[pix];
    w.q1 = off[pix + 1];
    // the line's nodes are sorted, so the reference's counting loop stops at
    // the first node >= py, the lower bound of py
    const uint32_t *voff = sv.voff + H.vline;
    const double *vn = sv.vnodes + H.vnode;
    uint32_t lo = voff[xo + 1], hi = voff[xo + 2];
    const uint32_t first = lo;
    while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (vn[mid] < (double)py) lo = mid + 1;
        else hi = mid;
    }
    w.odd = (lo - first) & 1u;
    return 2;
}

// Whether edge a -> b flips the point's parity: its crossing abscissa lies in
// [px, right]. Every operand is a float, so the reference evaluates it in FP32,
// one rounding per operation.
__device__ __forceinline__ bool edge_flips(float2 a, float2 b, float px, float py, float right) {
    if ((a.y >= py) == (b.y >= py)) return false;
    const float ix =
        __fadd_rn(__fdiv_rn(__fmul_rn(__fsub_rn(b.x, a.x), __fsub_rn(py, a.y)), __fsub_rn(b.y, a.y)), a.x);
    return px <= ix && ix <= right;
}

__device__ bool contain_point(const StoreView &sv, const PolyHdr &H, float px, float py) {
    PointPixel w;
    const int c = point_pixel(sv, H, px, py, w);
    if (c < 2) return c != 0;
    const uint2 *seq = sv.seq + H.seq;
    const float2 *r = sv.ring + H.ring;
    bool ret = w.odd;
#pragma unroll 1
    for (uint32_t q = w.q0; q < w.q1; q++) {
        const uint2 sq = seq[q];
#pragma unroll 1
        for (uint32_t k = 0; k < sq.y; k++)
            if (edge_flips(r[sq.x + k], r[sq.x + k + 1], px, py, w.right)) ret = !ret;
    }
    return ret;
}

// A point per lane up to its pixel; the BORDER pixels' sequences and their
// edges are flattened over the lanes, as a pixel lists from a few to hundreds
// of them and a warp would wait for its longest. 1M points in polygons of up to
// 5,000 vertices: 0.58 ms with a point's edges by its own lane, 0.19 ms so.
constexpr int kPointWarps = 8;
__global__ void __launch_bounds__(32 * kPointWarps)
    k_contain_points(const StoreView sv, uint64_t side_base, const float2 *__restrict__ pts,
                     const uint32_t *__restrict__ pairs, uint64_t n, uint8_t *__restrict__ out,
                     ContainCounters *__restrict__ ctr) {
    __shared__ float4 s_pt[kPointWarps][32];            // point, right border
    __shared__ const float2 *s_ring[kPointWarps][32];
    __shared__ uint32_t s_flip[kPointWarps][32];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    unsigned long long mine = 0;
#pragma unroll 1
    for (uint64_t k0 = (uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u); k0 < n;
         k0 += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t k = k0 + lane;
        int v = 0;
        PointPixel w{0u, 0u, 0.f, false};
        const uint2 *seq = nullptr;
        if (k < n) {
            const uint2 pq = load_pair(pairs, k);
            const PolyHdr &H = sv.hdr[side_base + pq.x];
            if (H.err) {
                v = 3;
            } else {
                const float2 P = pts[pq.y];
                v = point_pixel(sv, H, P.x, P.y, w);
                seq = sv.seq + H.seq + w.q0;
                s_pt[wib][lane] = make_float4(P.x, P.y, w.right, 0.f);
                s_ring[wib][lane] = sv.ring + H.ring;
            }
        }
        s_flip[wib][lane] = w.odd ? 1u : 0u;
        __syncwarp();
        uint32_t tsq;
        const uint32_t xsq = warp_excl_scan(w.q1 - w.q0, lane, tsq);
#pragma unroll 1
        for (uint32_t s0 = 0; s0 < tsq; s0 += 32) {
            const uint32_t si = s0 + lane;
            const int ow = warp_owner(xsq, si);
            const uint2 *q = reinterpret_cast<const uint2 *>(
                                 __shfl_sync(full, reinterpret_cast<unsigned long long>(seq), ow)) +
                             (si - __shfl_sync(full, xsq, ow));
            const uint2 sq = si < tsq ? *q : make_uint2(0u, 0u);
            uint32_t te;
            const uint32_t xe = warp_excl_scan(sq.y, lane, te);
#pragma unroll 1
            for (uint32_t e0 = 0; e0 < te; e0 += 32) {
                const uint32_t e = e0 + lane;
                const int oe = warp_owner(xe, e);
                const uint32_t f = __shfl_sync(full, sq.x, oe) + (e - __shfl_sync(full, xe, oe));
                const int c = __shfl_sync(full, ow, oe);
                if (e < te) {
                    const float4 p = s_pt[wib][c];
                    const float2 *r = s_ring[wib][c] + f;
                    if (edge_flips(r[0], r[1], p.x, p.y, p.z)) atomicXor(&s_flip[wib][c], 1u);
                }
            }
        }
        __syncwarp();
        if (k < n) {
            const bool in = v == 1 || (v == 2 && s_flip[wib][lane]);
            out[k] = v == 3 ? 2 : (in ? 1 : 0);
            mine += in;
        }
        __syncwarp();
    }
    for (int o = 16; o; o >>= 1) mine += __shfl_xor_sync(full, mine, o);
    if (lane == 0 && mine) atomicAdd(&ctr->found, mine);
}

// A target pixel's edges against the border of source pixel box (b0, b1, b2, b3)
// (the five float corners Ideal.cpp:1196-1200 builds): true on any crossing.
// Lanes take the pixel's edges, flattened over its sequences by a warp scan.
__device__ bool edges_cross_box(const StoreView &sv, const PolyHdr &T, uint32_t pb, double b0, double b1, double b2,
                                double b3, unsigned long long &tests) {
    const int lane = threadIdx.x & 31;
    const float2 c0 = make_float2((float)b0, (float)b1), c1 = make_float2((float)b0, (float)b3);
    const float2 c2 = make_float2((float)b2, (float)b3), c3 = make_float2((float)b2, (float)b1);
    const uint32_t *to = sv.offset + T.off;
    const uint2 *tseq = sv.seq + T.seq;
    const float2 *tr = sv.ring + T.ring;
    const uint32_t q0 = to[pb], q1 = to[pb + 1];
#pragma unroll 1
    for (uint32_t g = q0; g < q1; g += 32) {
        const uint32_t k = g + lane;
        const uint2 r = k < q1 ? tseq[k] : make_uint2(0u, 0u);
        uint32_t total;
        const uint32_t excl = warp_excl_scan(r.y, lane, total);
#pragma unroll 1
        for (uint32_t sb = 0; sb < total; sb += 32) {
            const uint32_t f = sb + lane;
            bool hit = false;
            const int owner = warp_owner(excl, f);
            const uint32_t ostart = __shfl_sync(0xffffffffu, r.x, owner);
            const uint32_t oex = __shfl_sync(0xffffffffu, excl, owner);
            if (f < total) {
                const float2 a = tr[ostart + (f - oex)], b = tr[ostart + (f - oex) + 1];
                hit = seg_intersect(a, b, c0, c1) || seg_intersect(a, b, c1, c2) || seg_intersect(a, b, c2, c3) ||
                      seg_intersect(a, b, c3, c0);
                tests += 4;
            }
            if (__any_sync(0xffffffffu, hit)) return true;
        }
    }
    return false;
}

// An entry of the queue: source pixel, target pixel; kOutBorder marks an OUT
// source pixel over a BORDER target pixel (the others are BORDER x BORDER).
constexpr uint32_t kOutBorder = 0x80000000u;

// Whether pixel pair e says "no"; part / nparts as in refine_pixel_pair.
__device__ __forceinline__ bool pixel_pair_violates(const StoreView &sv, const PolyHdr &S, const PolyHdr &T, uint2 e,
                                                    float4 *tb, unsigned long long &tests, uint32_t part,
                                                    uint32_t nparts) {
    if (!(e.x & kOutBorder)) return refine_pixel_pair(sv, S, T, e.x, e.y, tb, tests, part, nparts);
    if (part) return false;
    const int i = (int)((e.x & ~kOutBorder) % (uint32_t)S.dimx), j = (int)((e.x & ~kOutBorder) / (uint32_t)S.dimx);
    return edges_cross_box(sv, T, e.y, S.mbr[0] + i * S.step_x, S.mbr[1] + j * S.step_y,
                           S.mbr[0] + (i + 1) * S.step_x, S.mbr[1] + (j + 1) * S.step_y, tests);
}

// One warp per candidate pair up to its budget; what is left of a pair goes to
// k_contain_spill. A pair's result is written here as if no spilled pixel pair
// said "no".
__global__ void __launch_bounds__(kContainWarps * 32)
    k_contain(const StoreView sv, const uint32_t *__restrict__ pairs, uint64_t n, uint64_t tgt_base,
              unsigned long long *__restrict__ next, uint8_t *__restrict__ out, ContainCounters *__restrict__ ctr,
              SpillPool sp) {
    __shared__ uint2 queue[kContainWarps][kQueue];
    __shared__ float4 tbufs[kContainWarps][2 * kStage];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    uint2 *q = queue[wib];
    float4 *tb = tbufs[wib];
    const int cc = sv.category_count;
    unsigned long long my_found = 0, my_pp = 0, my_tests = 0;
    for (;;) {
        unsigned long long pid = 0;
        if (lane == 0) pid = atomicAdd(next, 1ull);
        pid = __shfl_sync(full, pid, 0);
        if (pid >= n) break;
        const uint32_t s = pairs[2 * pid], t = pairs[2 * pid + 1];
        const PolyHdr &S = sv.hdr[s];
        const PolyHdr &T = sv.hdr[tgt_base + t];
        if (S.err || T.err) {
            if (lane == 0) out[pid] = 2;
            continue;
        }
        // box::contain(box) (Box.cpp:59-64) of the MBRs
        if (!(T.mbr[0] >= S.mbr[0] && T.mbr[2] <= S.mbr[2] && T.mbr[1] >= S.mbr[1] && T.mbr[3] <= S.mbr[3])) {
            if (lane == 0) out[pid] = 0;
            continue;
        }
        const uint8_t *sst = sv.status + S.st, *tst = sv.status + T.st;
        const Window w = retrieve(S.mbr, S.step_x, S.step_y, S.dimx, S.dimy, T.mbr[0], T.mbr[1], T.mbr[2], T.mbr[3]);
        const int wh = w.ey - w.sy + 1;
        const long nw = (w.ex >= w.sx && w.ey >= w.sy) ? (long)(w.ex - w.sx + 1) * wh : 0;
        // the window's OUT and IN counts
        long n_out = 0, n_in = 0;
#pragma unroll 1
        for (long base = 0; base < nw; base += 32) {
            const long k = base + lane;
            int st = 1;
            if (k < nw) st = show_status(sst[(w.sy + (int)(k % wh)) * S.dimx + w.sx + (int)(k / wh)], cc);
            n_out += __popc(__ballot_sync(full, k < nw && st == 0));
            n_in += __popc(__ballot_sync(full, k < nw && st == 2));
        }
        int result;
        bool spilled = false;
        uint32_t head = 0;
        if (n_out == nw) {
            result = 0;
        } else if (n_in == nw) {
            result = 1;
        } else {
            bool violated = false, may_spill = sp.cap > 0;
            const float pp_cost = pixel_pair_cost(S, T);
            float spent = 0.f;
            int qn = 0;
            // one source window pixel per lane (x outer, y inner; IN pixels are
            // skipped), its target window flattened across the warp
            long base = 0;
            int tw_sx = 0, tw_sy = 0, tw_ey = -1, pa_st = 2;
            uint32_t pa = 0, excl = 0, total = 0, f = 0;
#pragma unroll 1
            for (bool more = true; more && !violated;) {
                while (qn + 32 <= kQueue) {
                    if (f >= total) {
                        if (base >= nw) {
                            more = false;
                            break;
                        }
                        const long k = base + lane;
                        uint32_t cnt = 0;
                        pa_st = 2;
                        if (k < nw) {
                            const int i = w.sx + (int)(k / wh), j = w.sy + (int)(k % wh);
                            pa = (uint32_t)(j * S.dimx + i);
                            pa_st = show_status(sst[pa], cc);
                            if (pa_st != 2) {
                                const double b0 = S.mbr[0] + i * S.step_x, b1 = S.mbr[1] + j * S.step_y;
                                const double b2 = S.mbr[0] + (i + 1) * S.step_x, b3 = S.mbr[1] + (j + 1) * S.step_y;
                                const Window tw = retrieve(T.mbr, T.step_x, T.step_y, T.dimx, T.dimy, b0, b1, b2, b3);
                                if (tw.ex >= tw.sx && tw.ey >= tw.sy) {
                                    tw_sx = tw.sx;
                                    tw_sy = tw.sy;
                                    tw_ey = tw.ey;
                                    cnt = (uint32_t)((tw.ex - tw.sx + 1) * (tw.ey - tw.sy + 1));
                                }
                            }
                        }
                        excl = warp_excl_scan(cnt, lane, total);
                        base += 32;
                        f = 0;
                        continue;
                    }
                    const uint32_t item = f + lane;
                    f += 32;
                    const int owner = warp_owner(excl, item);
                    const uint32_t o_excl = __shfl_sync(full, excl, owner);
                    const int o_sx = __shfl_sync(full, tw_sx, owner);
                    const int o_sy = __shfl_sync(full, tw_sy, owner);
                    const int o_ey = __shfl_sync(full, tw_ey, owner);
                    const int o_st = __shfl_sync(full, pa_st, owner);
                    const uint32_t o_pa = __shfl_sync(full, pa, owner);
                    bool out_in = false, edges = false;
                    uint32_t pb = 0;
                    if (item < total) {
                        const uint32_t r = item - o_excl;
                        const int th = o_ey - o_sy + 1;
                        const int u = o_sx + (int)(r / (uint32_t)th), v = o_sy + (int)(r % (uint32_t)th);
                        pb = (uint32_t)(v * T.dimx + u);
                        const int pb_st = show_status(tst[pb], cc);
                        out_in = o_st == 0 && pb_st == 2;
                        edges = pb_st == 1;  // the source pixel is OUT or BORDER
                    }
                    if (__any_sync(full, out_in)) {
                        violated = true;
                        break;
                    }
                    const unsigned m = __ballot_sync(full, edges);
                    if (edges) q[qn + __popc(m & ((1u << lane) - 1))] = make_uint2(o_pa | (o_st == 0 ? kOutBorder : 0u), pb);
                    qn += __popc(m);
                }
                if (violated || qn == 0) continue;
                __syncwarp();
#pragma unroll 1
                for (int k = 0; k < qn && !violated; k++) {
                    if (may_spill && spent > sp.budget) {
                        if (spill_rest(sp, pid, q, k, qn, pp_cost, lane, &head, &spilled)) {
                            if (lane == 0) my_pp += qn - k;
                            break;
                        }
                        may_spill = false;  // the pool is full
                    }
                    if (lane == 0) my_pp++;
                    violated = pixel_pair_violates(sv, S, T, q[k], tb, my_tests, 0, 1);
                    spent += pp_cost;
                }
                qn = 0;
                __syncwarp();
            }
            if (violated) {
                result = 0;
            } else {
                // t's first vertex (Ideal.cpp:1228-1230)
                bool in = false;
                if (lane == 0) {
                    const float2 p0 = sv.ring[T.ring];
                    in = contain_point(sv, S, p0.x, p0.y);
                }
                result = __shfl_sync(full, in, 0) ? 1 : 0;
            }
        }
        if (lane == 0) {
            out[pid] = (uint8_t)result;
            my_found += result == 1;
            if (spilled && result == 0) sp.flag[head] = 1u;  // nothing left to find out
        }
        __syncwarp();
    }
    for (int o = 16; o; o >>= 1) my_tests += __shfl_xor_sync(full, my_tests, o);
    if (lane == 0) {
        atomicAdd(&ctr->found, my_found);
        atomicAdd(&ctr->pixel_pairs, my_pp);
        atomicAdd(&ctr->segment_tests, my_tests);
    }
}

// The pixel pairs that k_contain spilled, over all warps: a "no" takes back
// the result that k_contain wrote (1, or the pair's flag were set).
__global__ void __launch_bounds__(kContainWarps * 32, 3)
    k_contain_spill(const StoreView sv, const uint32_t *__restrict__ pairs, uint64_t tgt_base, SpillPool sp,
                    uint8_t *__restrict__ out, ContainCounters *__restrict__ ctr) {
    __shared__ float4 tbufs[kContainWarps][2 * kStage];
    float4 *tb = tbufs[threadIdx.x >> 5];
    unsigned long long lost = 0, my_tests = 0;
    spill_units(
        sp,
        [&](unsigned long long p, uint2 e, uint32_t part, uint32_t nparts) {
            const PolyHdr &S = sv.hdr[pairs[2 * p]];
            const PolyHdr &T = sv.hdr[tgt_base + pairs[2 * p + 1]];
            return pixel_pair_violates(sv, S, T, e, tb, my_tests, part, nparts);
        },
        [&](unsigned long long p) {
            out[p] = 0;
            lost++;
        });
    for (int o = 16; o; o >>= 1) my_tests += __shfl_xor_sync(0xffffffffu, my_tests, o);
    if ((threadIdx.x & 31) == 0) {
        if (lost) atomicAdd(&ctr->found, 0ull - lost);
        if (my_tests) atomicAdd(&ctr->segment_tests, my_tests);
    }
}

}  // namespace

}  // namespace farm

using namespace farm;

extern "C" int farm_contain(farm_store *s, const uint32_t *pairs, uint64_t n, int mem, uint8_t *out, uint64_t *found,
                            farm_stats *st) {
    if (!s || (n && (!pairs || !out))) {
        set_error("invalid arguments to farm_contain");
        return FARM_EINVAL;
    }
    if (!s->rasterized) {
        set_error("farm_contain: rasterize first");
        return FARM_EINVAL;
    }
    if (s->n_side[1] == 0) {
        set_error("farm_contain: no target side loaded");
        return FARM_EINVAL;
    }
    FARM_TRY(check_pairs(s, pairs, n, mem, false, "farm_contain"));
    cudaStream_t stream = s->stream;
    const uint32_t *dpairs = pairs;
    uint8_t *dout = out;
    if (mem == FARM_MEM_HOST && n) {
        FARM_TRY(s->d_pairs.ensure(8 * n));
        FARM_CUDA(cudaMemcpyAsync(s->d_pairs.p, pairs, 8 * n, cudaMemcpyHostToDevice, stream));
        dpairs = s->d_pairs.as<uint32_t>();
        FARM_TRY(s->d_out.ensure(n + 16));
        dout = s->d_out.as<uint8_t>();
    }
    FARM_TRY(s->d_counters.ensure(256));
    unsigned long long *next = s->d_counters.as<unsigned long long>();
    ContainCounters *ctr = reinterpret_cast<ContainCounters *>(next + 1);
    static_assert(8 + sizeof(ContainCounters) <= 64, "the spill counters follow at [8]");
    FARM_CUDA(cudaMemsetAsync(next, 0, 88, stream));
    SpillPool sp;
    if (n) FARM_TRY(spill_pool(s, n, next + 8, 512.f, 4096.f, &sp));
    FARM_CUDA(cudaEventRecord(s->ev[6], stream));
    if (n) {
        const uint64_t most = (uint64_t)sm_count() * 8;
        k_contain<<<(unsigned)(n < most ? n : most), kContainWarps * 32, 0, stream>>>(s->view(), dpairs, n,
                                                                                      s->n_side[0], next, dout, ctr, sp);
        k_contain_spill<<<3 * sm_count(), kContainWarps * 32, 0, stream>>>(s->view(), dpairs, s->n_side[0], sp, dout,
                                                                           ctr);
        FARM_CUDA(cudaGetLastError());
        s->launches += 2;
    }
    FARM_CUDA(cudaEventRecord(s->ev[7], stream));
    ContainCounters h{};
    FARM_CUDA(cudaMemcpyAsync(&h, ctr, sizeof h, cudaMemcpyDeviceToHost, stream));
    if (mem == FARM_MEM_HOST && n) FARM_CUDA(cudaMemcpyAsync(out, dout, n, cudaMemcpyDeviceToHost, stream));
    FARM_CUDA(cudaStreamSynchronize(stream));
    if (found) *found = h.found;
    if (st) {
        memset(st, 0, sizeof *st);
        st->pairs = n;
        st->found = h.found;
        st->border_pairs = h.pixel_pairs;
        st->segment_tests = h.segment_tests;
        float ms = 0;
        cudaEventElapsedTime(&ms, s->ev[6], s->ev[7]);
        st->ms_total = ms;
        st->ms_stage[2] = ms;
        st->kernel_launches = n ? 2 : 0;
    }
    return FARM_OK;
}

extern "C" int farm_contain_points(farm_store *s, int side, const float *xy, uint64_t npoints, const uint32_t *pairs,
                                   uint64_t n, int mem, uint8_t *out, uint64_t *found) {
    if (!s || side < 0 || side > 1 || (n && (!pairs || !out || !xy))) {
        set_error("invalid arguments to farm_contain_points");
        return FARM_EINVAL;
    }
    if (!s->rasterized) {
        set_error("farm_contain_points: rasterize first");
        return FARM_EINVAL;
    }
    FARM_TRY(check_pair_limits(s, pairs, n, mem, s->n_side[side], npoints, "farm_contain_points", "polygons",
                               "points"));
    if (mem == FARM_MEM_DEVICE && n && (reinterpret_cast<uintptr_t>(xy) & 7u)) {
        // the kernel reads whole (x, y) pairs: 8-byte loads
        set_error("farm_contain_points: device points must start on an 8-byte boundary");
        return FARM_EINVAL;
    }
    cudaStream_t stream = s->stream;
    const uint32_t *dpairs = pairs;
    const float2 *dpts = reinterpret_cast<const float2 *>(xy);
    uint8_t *dout = out;
    if (mem == FARM_MEM_HOST && n) {
        FARM_TRY(s->d_pairs.ensure(8 * n));
        FARM_CUDA(cudaMemcpyAsync(s->d_pairs.p, pairs, 8 * n, cudaMemcpyHostToDevice, stream));
        dpairs = s->d_pairs.as<uint32_t>();
        FARM_TRY(s->d_points.ensure(8 * npoints + 16));
        FARM_CUDA(cudaMemcpyAsync(s->d_points.p, xy, 8 * npoints, cudaMemcpyHostToDevice, stream));
        dpts = s->d_points.as<float2>();
        FARM_TRY(s->d_out.ensure(n + 16));
        dout = s->d_out.as<uint8_t>();
    }
    FARM_TRY(s->d_counters.ensure(256));
    ContainCounters *ctr = reinterpret_cast<ContainCounters *>(s->d_counters.as<unsigned long long>() + 1);
    FARM_CUDA(cudaMemsetAsync(ctr, 0, sizeof(ContainCounters), stream));
    if (n) {
        unsigned blocks = grid_for(n, 256);
        if (blocks > 16u * (unsigned)sm_count()) blocks = 16u * (unsigned)sm_count();
        k_contain_points<<<blocks, 256, 0, stream>>>(s->view(), side == 0 ? 0 : s->n_side[0], dpts, dpairs, n, dout,
                                                     ctr);
        FARM_CUDA(cudaGetLastError());
        s->launches++;
    }
    ContainCounters h{};
    FARM_CUDA(cudaMemcpyAsync(&h, ctr, sizeof h, cudaMemcpyDeviceToHost, stream));
    if (mem == FARM_MEM_HOST && n) FARM_CUDA(cudaMemcpyAsync(out, dout, n, cudaMemcpyDeviceToHost, stream));
    FARM_CUDA(cudaStreamSynchronize(stream));
    if (found) *found = h.found;
    return FARM_OK;
}
