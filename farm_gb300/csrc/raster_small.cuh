// Small polygons rasterized whole, a block per polygon (included by raster.cu).
//
// The flattened pipeline (raster_chunk) takes about 150 launches and a dozen
// waits whatever its input, and passes every intermediate through memory: for
// a few hundred polygons it is all latency, for ten thousand of a few hundred
// vertices mostly. Here one block takes a polygon through phase 2 from the
// walk to the cell areas, with barriers where the pipeline has launches: the
// same walk and clip code, the same orders (stable bucketing by one warp,
// points of a column in clip order), so the same bytes. Its intermediates lie
// in a scratch slice per block, which stays in L1/L2.
//
// 11,000 polygons of 16..1,024 vertices (configuration 1): phase 2 took
// 3.3 ms of device time and 160 launches, 1.5 ms and a dozen so.
//
// Loops are not unrolled: most run once or twice per thread, and what the
// warps wait for then is instruction fetch (kernels of 96 and 88 KB unrolled,
// 66 and 63 KB so: 3.17 -> 2.96 ms for that join as a whole).
#pragma once

// Two kernels: the walk (sequences, nodes) needs 128 registers a thread, the
// rest half of them, so that twice the blocks are resident. Blocks of 64
// threads while there are polygons to fill the chip with them (most of 16 to
// 1,024 vertices have little for more), of 256 for few polygons, whose largest
// one is then the whole wait.
constexpr uint32_t kSmallMany = 1024;  // polygons from which the narrow blocks are taken
constexpr int kWalkBlocks64 = 8, kFillBlocks64 = 14, kBlocks256 = 2;  // resident per SM
// A polygon is small up to these sizes (twice the edges and nodes for blocks of
// 256 threads): above them a block alone is slower than the pipeline's whole
// chip, and the shared counters would not fit. Joins of 400 polygons of up to
// 4,000 vertices 2.19 ms so, 2.79 ms by the pipeline; 1,000 at -v 64 3.05 / 4.02;
// 10,000 of up to 2,000 4.32 / 6.64.
constexpr uint32_t kSmallBig = 256;  // edges from which a small polygon is taken first
constexpr uint32_t kSmallEdges = 2048, kSmallNodes = 8192, kSmallPix = 2048, kSmallLines = 512;

// What the host needs to know of phase 1 (one copy): array totals, and the
// small polygons' number and largest sizes, which size the scratch.
struct SmallInfo {
    unsigned long long seq, hnodes, vnodes;  // totals over all polygons
    unsigned long long n, big, rest;         // small polygons: all, those taken first, the others
    unsigned long long next[2];              // the kernels' next polygons
    unsigned long long edges, cross, hn, vn, pix, lines;  // their largest
    unsigned long long left;                 // small polygons left to the pipeline (scratch too short)
    unsigned long long clip_x, clip_y, crossings;         // points and crossings of the small polygons
};

struct SmallArgs {
    StoreView sv;
    PolyHdr *hdr;
    const WalkF *wf;
    const uint32_t *list;
    const uint64_t *off;
    const uint16_t *c16;
    uint64_t ne_all;
    const double *colx, *rowy;
    const LineF *colf, *rowf;
    uint8_t *status;
    uint32_t *offset, *hoff, *voff;
    uint2 *seq;
    double *hnodes, *vnodes, *areas;
    uint8_t *done;
    SmallInfo *info;
    unsigned char *scratch;
    uint64_t slice;  // scratch bytes per block
    uint32_t cap_e, cap_c, cap_h, cap_v, cap_x, cap_cp, cap_y, hash;
    uint32_t pix, lines;  // shared counters
    uint32_t n, big, npoly;
    int cert, cc;
};

// The scratch slice's arrays. The crossings and the unsorted nodes are done
// with when the cell clip's points are written in their place.
struct SmallScratch {
    uint32_t *cf, *ct, *ce, *hl, *vl, *we;
    uint64_t *wa;
    double *hv, *vv;
    uint32_t *xc, *sc, *tab;
    float2 *xp, *sp;
    uint8_t *drop;
    float2 *cp;
    uint32_t *cpc;
    uint32_t *yr;
    float2 *yp, *ys;
};
__host__ __device__ inline uint64_t small_scratch(const SmallArgs &a, unsigned char *base, SmallScratch *s) {
    uint64_t at = 0;
    auto take = [&](uint64_t bytes) {
        unsigned char *p = base + at;
        at += (bytes + 15) & ~15ull;
        return p;
    };
    SmallScratch d;
    d.hv = reinterpret_cast<double *>(take(8ull * a.cap_h));
    d.vv = reinterpret_cast<double *>(take(8ull * a.cap_v));
    d.wa = reinterpret_cast<uint64_t *>(take(8ull * a.cap_e));
    d.we = reinterpret_cast<uint32_t *>(take(4ull * a.cap_e));
    d.hl = reinterpret_cast<uint32_t *>(take(4ull * a.cap_h));
    d.vl = reinterpret_cast<uint32_t *>(take(4ull * a.cap_v));
    d.cf = reinterpret_cast<uint32_t *>(take(4ull * a.cap_c));
    d.ct = reinterpret_cast<uint32_t *>(take(4ull * a.cap_c));
    d.ce = reinterpret_cast<uint32_t *>(take(4ull * a.cap_c));
    const uint64_t first = at;
    at = 0;
    d.yp = reinterpret_cast<float2 *>(take(8ull * a.cap_y));
    d.ys = reinterpret_cast<float2 *>(take(8ull * a.cap_y));
    d.yr = reinterpret_cast<uint32_t *>(take(4ull * a.cap_y));
    if (at < first) at = first;
    d.xp = reinterpret_cast<float2 *>(take(8ull * a.cap_x));
    d.sp = reinterpret_cast<float2 *>(take(8ull * a.cap_x));
    d.xc = reinterpret_cast<uint32_t *>(take(4ull * a.cap_x));
    d.sc = reinterpret_cast<uint32_t *>(take(4ull * a.cap_x));
    d.tab = reinterpret_cast<uint32_t *>(take(4ull * a.hash));
    d.drop = take(a.cap_x);
    d.cp = reinterpret_cast<float2 *>(take(8ull * a.cap_cp));
    d.cpc = reinterpret_cast<uint32_t *>(take(4ull * a.cap_cp));
    if (s) *s = d;
    return (at + 255) & ~255ull;
}

// Phase 1's totals per polygon into sizes already scanned (k_set_node_bases'
// work), and the pick of the small polygons.
__global__ void k_small_pick(PolyHdr *__restrict__ hdr, uint32_t npoly, const uint64_t *__restrict__ sz,
                             const uint64_t *__restrict__ sc, const uint64_t *__restrict__ off, int counts_ok,
                             const int *__restrict__ ovf, uint32_t *__restrict__ list, uint8_t *__restrict__ done,
                             SmallInfo *__restrict__ info) {
    const uint64_t n1 = (uint64_t)npoly + 1;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        info->seq = sc[npoly];
        info->hnodes = sc[n1 + npoly];
        info->vnodes = sc[2 * n1 + npoly];
    }
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t wide = npoly < kSmallMany ? 2 : 1;  // blocks of 256 threads
#pragma unroll 1
    for (uint32_t p0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; p0 < npoly; p0 += gridDim.x * blockDim.x) {
        const uint32_t p = p0 + lane;
        bool small = false;
        uint32_t ne = 0, cross = 0, hn = 0, vn = 0, pix = 0, lines = 0;
        if (p < npoly) {
            PolyHdr &h = hdr[p];
            h.seq = sc[p];
            h.n_seq = (uint32_t)sz[p];
            h.hnode = sc[n1 + p];
            h.n_hnodes = (uint32_t)sz[n1 + p];
            h.vnode = sc[2 * n1 + p];
            h.n_vnodes = (uint32_t)sz[2 * n1 + p];
            const uint64_t edges = off[p + 1] - off[p];
            lines = (uint32_t)(h.dimx > h.dimy ? h.dimx : h.dimy) + 3;
            small = counts_ok && *ovf == 0 && edges <= wide * kSmallEdges && sz[n1 + p] <= wide * kSmallNodes &&
                    sz[2 * n1 + p] <= wide * kSmallNodes && sz[p] <= 2 * wide * kSmallNodes && h.P <= kSmallPix &&
                    lines <= kSmallLines;
            done[p] = 0;
            ne = (uint32_t)edges;
            cross = h.n_seq;
            hn = h.n_hnodes;
            vn = h.n_vnodes;
            pix = h.P;
        }
        // the list from the front: larger polygons, from the back: the others
        const unsigned any = __ballot_sync(full, small), front = __ballot_sync(full, small && ne >= kSmallBig);
        if (!any) continue;
        unsigned long long at_f = 0;
        if (lane == 0) {
            at_f = atomicAdd(&info->big, (unsigned long long)__popc(front));
            atomicAdd(&info->n, (unsigned long long)__popc(any));
        }
        at_f = __shfl_sync(full, at_f, 0);
        const unsigned back = any & ~front;
        unsigned long long at_k = 0;
        if (lane == 0 && back) at_k = atomicAdd(&info->rest, (unsigned long long)__popc(back));
        at_k = __shfl_sync(full, at_k, 0);
        const unsigned below = (1u << lane) - 1u;
        if (small) {
            if (ne >= kSmallBig) list[at_f + __popc(front & below)] = p;
            else list[npoly - 1 - (at_k + __popc(back & below))] = p;
        }
        auto largest = [&](unsigned long long *to, uint32_t v) {
            const uint32_t m = __reduce_max_sync(full, small ? v : 0u);
            if (lane == 0) atomicMax(to, (unsigned long long)m);
        };
        largest(&info->edges, ne);
        largest(&info->cross, cross);
        largest(&info->hn, hn);
        largest(&info->vn, vn);
        largest(&info->pix, pix);
        largest(&info->lines, lines);
    }
}

// The next polygon of a kernel, largest ones first: ~0 past the last.
__device__ __forceinline__ uint32_t small_next(const SmallArgs &a, int which, uint32_t *shared) {
    __syncthreads();  // the last polygon's shared arrays are done with
    if (threadIdx.x == 0) {
        const unsigned long long q = atomicAdd(&a.info->next[which], 1ull);
        *shared = q >= a.n ? ~0u : (q < a.big ? a.list[q] : a.list[a.npoly - 1 - (q - a.big)]);
    }
    __syncthreads();
    return *shared;
}

// exclusive scan over the block (several small counts may be packed in one
// word); total of the block in *total
template <int NT>
__device__ __forceinline__ uint64_t small_scan(uint64_t v, uint64_t *sums, uint64_t *total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint64_t incl = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint64_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    __syncthreads();  // sums free again
    if (lane == 31) sums[w] = incl;
    __syncthreads();
    uint64_t base = 0, all = 0;
#pragma unroll
    for (int k = 0; k < NT / 32; k++) {
        if (k < w) base += sums[k];
        all += sums[k];
    }
    *total = all;
    return base + incl - v;
}

// counts c[0, n) to their exclusive prefix sums, c[n] the total
template <int NT>
__device__ void small_prefix(uint32_t *c, uint32_t n, uint64_t *sums) {
    uint64_t run = 0;
    __syncthreads();
#pragma unroll 1
    for (uint32_t b = 0; b < n; b += NT) {
        const uint32_t i = b + threadIdx.x;
        const uint64_t v = i < n ? c[i] : 0u;
        uint64_t total;
        const uint64_t ex = small_scan<NT>(v, sums, &total);
        if (i < n) c[i] = (uint32_t)(run + ex);
        run += total;
    }
    if (threadIdx.x == 0) c[n] = (uint32_t)run;
    __syncthreads();
}

struct SmallSink {
    static constexpr bool kValues = true;
    int dimx, dimy;
    uint32_t edge, c, hn, vn;
    uint32_t *cf, *ct, *ce, *hl, *vl;
    double *hv, *vv;
    bool bad = false;
    __device__ bool inb(int x, int y) const { return x >= 0 && x < dimx && y >= 0 && y < dimy; }
    __device__ void border(int x, int y) {
        if (!inb(x, y)) bad = true;
    }
    __device__ void cross(int fx, int fy, int tx, int ty) {
        if (!inb(fx, fy) || !inb(tx, ty)) {
            bad = true;
            return;
        }
        cf[c] = (uint32_t)(fy * dimx + fx);
        ct[c] = (uint32_t)(ty * dimx + tx);
        ce[c] = edge;
        c++;
    }
    __device__ void hnode(int line, double v) {
        if (line < 0 || line > dimy + 1) { bad = true; return; }
        hl[hn] = (uint32_t)line;
        hv[hn] = v;
        hn++;
    }
    __device__ void vnode(int line, double v) {
        if (line < 0 || line > dimx + 1) { bad = true; return; }
        vl[vn] = (uint32_t)line;
        vv[vn] = v;
        vn++;
    }
    __device__ void fail() { bad = true; }
    __device__ bool failed() const { return bad; }
};

// A line's n nodes sorted in place by one warp (as k_line_sort_warp / _mid:
// a bitonic network on order-preserving keys).
__device__ void small_sort_line(double *v, uint32_t n, uint64_t *buf, int lane) {
    if (n < 2) return;
    if (n <= 32) {
        uint64_t k = (uint32_t)lane < n ? dkey(v[lane]) : ~0ull;
#pragma unroll 1
        for (int size = 2; size <= 32; size <<= 1)
#pragma unroll 1
            for (int j = size >> 1; j > 0; j >>= 1) {
                const uint64_t o = __shfl_xor_sync(0xffffffffu, k, j);
                const bool up = (lane & size) == 0, lower = (lane & j) == 0;
                k = (lower == up) ? (k < o ? k : o) : (k < o ? o : k);
            }
        if ((uint32_t)lane < n) v[lane] = dval(k);
        return;
    }
    // over kLineMid the network runs on the keys in place: elements past n
    // count as the largest key and never move below it
    const bool sm = n <= (uint32_t)kLineMid;
    uint64_t *key = sm ? buf : reinterpret_cast<uint64_t *>(v);
    uint32_t N = 64;
    while (N < n) N <<= 1;
#pragma unroll 1
    for (uint32_t i = lane; i < n; i += 32) key[i] = dkey(v[i]);
    if (sm)
#pragma unroll 1
        for (uint32_t i = n + lane; i < N; i += 32) key[i] = ~0ull;
    __syncwarp();
#pragma unroll 1
    for (uint32_t k = 2; k <= N; k <<= 1)
#pragma unroll 1
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
#pragma unroll 1
            for (uint32_t i = lane; i < N; i += 32) {
                // ascending runs only: the first step of a merge pairs i with its mirror
                const uint32_t ixj = j == (k >> 1) ? (i ^ (k - 1)) : (i ^ j);
                if (ixj > i && ixj < (sm ? N : n)) {
                    const uint64_t x = key[i], y = key[ixj];
                    if (x > y) {
                        key[i] = y;
                        key[ixj] = x;
                    }
                }
            }
            __syncwarp();
        }
#pragma unroll 1
    for (uint32_t i = lane; i < n; i += 32) v[i] = dval(key[i]);
    __syncwarp();
}

// Items [0, n) with buckets key(i) to their stable positions by one warp:
// cur[b * step] is bucket b's next position (its end afterwards).
template <typename Key, typename Put>
__device__ __forceinline__ void small_stable(uint32_t i0, uint32_t n, uint32_t *cur, uint32_t step, int lane, Key key,
                                             Put put) {
#pragma unroll 1
    for (uint32_t b = i0; b < n; b += 32) {
        const uint32_t i = b + lane;
        const unsigned act = __ballot_sync(0xffffffffu, i < n);
        if (i < n) {
            const uint32_t k = key(i);
            const unsigned grp = __match_any_sync(act, k);
            const uint32_t at = cur[k * step] + (uint32_t)__popc(grp & ((1u << lane) - 1u));
            put(i, at);
            __syncwarp(act);
            if (lane == __ffs(grp) - 1) cur[k * step] += (uint32_t)__popc(grp);
        }
        __syncwarp();
    }
}

// The same by the whole block, each warp its share of the items: counters per
// (bucket, warp) in cnt (nb x warps + 1), start[b] the buckets' starts (nb +
// 1). put may run in any order across warps; before(): run by all once the
// starts are known, ahead of any put.
template <int NT, typename Key, typename Put, typename Before>
__device__ __forceinline__ void small_bucket(uint32_t n, uint32_t nb, uint32_t *cnt, uint32_t *start, uint64_t *sums,
                                             Key key, Put put, Before before) {
    constexpr uint32_t W = NT / 32;
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
#pragma unroll 1
    for (uint32_t k = tid; k < nb * W; k += NT) cnt[k] = 0;
    __syncthreads();
    const uint32_t part = ((n + W - 1) / W + 31) & ~31u;
    const uint32_t i0 = min(n, warp * part), i1 = min(n, i0 + part);
#pragma unroll 1
    for (uint32_t i = i0 + (tid & 31); i < i1; i += 32) atomicAdd(&cnt[key(i) * W + warp], 1u);
    small_prefix<NT>(cnt, nb * W, sums);
#pragma unroll 1
    for (uint32_t b = tid; b <= nb; b += NT) start[b] = cnt[b * W];
    __syncthreads();
    before();
    small_stable(i0, i1, cnt + warp, W, (int)(tid & 31), key, put);
    __syncthreads();
}

// Walk, edge sequences and sorted grid-line nodes of the small polygons.
template <int NT, int kBlocks>
__global__ void __launch_bounds__(NT, kBlocks) k_small_walk(SmallArgs a) {
    extern __shared__ uint32_t sh[];
    constexpr int kWarps = NT / 32;
    const uint32_t most = a.pix > a.lines ? a.pix : a.lines;
    uint32_t *start = sh, *cnt = sh + most + 1;  // cnt: most x warps + 1
    uint32_t *linec = start;
    __shared__ uint64_t sums[kWarps];
    __shared__ uint64_t sortb[kWarps][kLineMid];
    __shared__ int s_err;
    __shared__ uint32_t s_next;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    SmallScratch s;
    small_scratch(a, a.scratch + blockIdx.x * a.slice, &s);
    for (;;) {
        const uint32_t p = small_next(a, 0, &s_next);
        if (p == ~0u) break;
        const PolyHdr &h = a.hdr[p];
        if (tid == 0) {
            s_err = h.err;
            a.done[p] = 1;
        }
        __syncthreads();
        if (s_err) {  // failed in phase 1: its offsets end in its (zero) sequence count
            if (tid == 0) a.offset[h.off + h.P] = h.n_seq;
            continue;
        }
        const uint64_t e0 = a.off[p];
        const uint32_t ne = (uint32_t)(a.off[p + 1] - e0);
        const float2 *r = a.sv.ring + h.ring;
        const int dimx = h.dimx, dimy = h.dimy;
        // ---- edge walk: crossings and nodes in edge order. The edges that
        // have any, fewer than half, are listed first, so that the lanes that
        // walk do so together. Packed: crossings, h-nodes, v-nodes, edges.
        uint64_t run = 0;
#pragma unroll 1
        for (uint32_t b = 0; b < ne; b += NT) {
            const uint32_t e = b + tid;
            uint64_t c = 0, total;
            if (e < ne) {
                c = (uint64_t)a.c16[e0 + e] | ((uint64_t)a.c16[a.ne_all + e0 + e] << 16) |
                    ((uint64_t)a.c16[2 * a.ne_all + e0 + e] << 32);
                if (c) c |= 1ull << 48;
            }
            const uint64_t at = run + small_scan<NT>(c, sums, &total);
            run += total;
            if (c) {
                s.we[at >> 48] = e;
                s.wa[at >> 48] = at;
            }
        }
        __syncthreads();
        const uint32_t nC = (uint32_t)(run & 0xFFFF), nH = (uint32_t)((run >> 16) & 0xFFFF),
                       nV = (uint32_t)((run >> 32) & 0xFFFF), nW = (uint32_t)(run >> 48);
#pragma unroll 1
        for (uint32_t i = tid; i < nW; i += NT) {
            const uint64_t at = s.wa[i];
            const uint32_t e = s.we[i];
            SmallSink k;
            k.dimx = dimx;
            k.dimy = dimy;
            k.edge = e;
            k.c = (uint32_t)(at & 0xFFFF);
            k.hn = (uint32_t)((at >> 16) & 0xFFFF);
            k.vn = (uint32_t)((at >> 32) & 0xFFFF);
            k.cf = s.cf;
            k.ct = s.ct;
            k.ce = s.ce;
            k.hl = s.hl;
            k.vl = s.vl;
            k.hv = s.hv;
            k.vv = s.vv;
            walk_edge(h, a.wf[p], r[e], r[e + 1], k);
        }
        __syncthreads();
        // ---- sequences (process_crosses): visit v enters pixel to[c], c the
        // crossing before it; the ring's last crossing comes first (k_visits)
        uint32_t *offs = a.offset + h.off;
        uint2 *seq = a.seq + h.seq;
        if (nC == 0) {  // one sequence covering the ring (Ideal.cpp:523-529)
#pragma unroll 1
            for (uint32_t i = tid; i < h.P; i += NT) offs[i] = i ? 1u : 0u;
            if (tid == 0) seq[0] = make_uint2(0u, h.nv);
        } else {
            const uint32_t wrap = s.ct[nC - 1];
#pragma unroll 1
            for (uint32_t c = tid; c < nC; c += NT)
                if (s.cf[c + 1 == nC ? 0 : c + 1] != s.ct[c]) atomicMin(&s_err, FARM_EASSERT);
            small_bucket<NT>(
                nC, h.P, cnt, start, sums, [&](uint32_t v) { return s.ct[v ? v - 1 : nC - 1]; },
                [&](uint32_t v, uint32_t at) {
                    if (v == 0) {  // add_edge(0, first leave) and add_edge(last enter, nv - 2)
                        const uint32_t ein = s.ce[nC - 1];
                        seq[at] = make_uint2(0u, s.ce[0] + 1u);
                        seq[at + 1] = make_uint2(ein, h.nv - 2u - ein + 1u);
                    } else {
                        const uint32_t ein = s.ce[v - 1], eout = s.ce[v];
                        if (eout < ein) atomicMin(&s_err, FARM_EASSERT);
                        seq[at + (at > start[wrap] ? 1u : 0u)] = make_uint2(ein, eout - ein + 1u);
                    }
                },
                [&]() {
#pragma unroll 1
                    for (uint32_t i = tid; i < h.P; i += NT) offs[i] = start[i] + (i > wrap ? 1u : 0u);
                });
        }
        if (tid == 0) offs[h.P] = h.n_seq;
        __syncthreads();
        // ---- grid-line nodes (process_intersection), horizontal then vertical
#pragma unroll 1
        for (int vert = 0; vert < 2; vert++) {
            const uint32_t n = vert ? nV : nH, dim = (uint32_t)(vert ? dimx : dimy);
            const uint32_t *line = vert ? s.vl : s.hl;
            const double *val = vert ? s.vv : s.hv;
            double *out = vert ? a.vnodes + h.vnode : a.hnodes + h.hnode;
            uint32_t *lo = vert ? a.voff + h.vline : a.hoff + h.hline;
#pragma unroll 1
            for (uint32_t i = tid; i <= dim + 2; i += NT) linec[i] = 0;
            __syncthreads();
#pragma unroll 1
            for (uint32_t i = tid; i < n; i += NT) atomicAdd(&linec[line[i]], 1u);
            small_prefix<NT>(linec, dim + 2, sums);
#pragma unroll 1
            for (uint32_t l = tid; l < dim + 2; l += NT) {
                const uint32_t st = linec[l];
                uint32_t v = linec[l + 1] != st ? st : 0u;
                if (l == dim || (vert && l == dim + 1)) v = n;
                lo[l] = v;
            }
            __syncthreads();
#pragma unroll 1
            for (uint32_t i = tid; i < n; i += NT) out[atomicAdd(&linec[line[i]], 1u)] = val[i];
            __syncthreads();  // linec[l] is now line l's end
#pragma unroll 1
            for (uint32_t l = warp; l < dim + 2; l += kWarps) {
                const uint32_t b = l ? linec[l - 1] : 0u;
                small_sort_line(out + b, linec[l] - b, sortb[warp], lane);
            }
            __syncthreads();
        }
        if (tid == 0) {
            if (s_err) atomicMin(&a.hdr[p].err, s_err);
            atomicAdd(&a.info->crossings, (unsigned long long)nC);
        }
    }
}

// Scanline, both clips, cell areas and classes of the small polygons.
template <int NT, int kBlocks>
__global__ void __launch_bounds__(NT, kBlocks) k_small_fill(SmallArgs a) {
    extern __shared__ uint32_t sh[];
    constexpr int kWarps = NT / 32;
    uint32_t *pixc = sh;                   // per pixel, pix + 1
    uint32_t *linec = pixc + a.pix + 1;    // first clip point of each column, lines + 1
    uint32_t *cpst = linec + a.lines + 1;  // column polygons, lines + 1
    uint32_t *yst = cpst + a.lines + 1;    // first cell point of each column, lines + 1
    uint32_t *cnt = yst + a.lines + 1;     // lines x warps + 1
    __shared__ uint64_t sums[kWarps];
    __shared__ int s_full;
    __shared__ uint32_t s_next;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    SmallScratch s;
    small_scratch(a, a.scratch + blockIdx.x * a.slice, &s);
    for (;;) {
        const uint32_t p = small_next(a, 1, &s_next);
        if (p == ~0u) break;
        const PolyHdr &h = a.hdr[p];
        if (h.err) continue;
        if (tid == 0) s_full = 0;
        __syncthreads();
        const float2 *r = a.sv.ring + h.ring;
        const uint32_t ne = h.nv - 1;  // stored vertices
        const int dimx = h.dimx, dimy = h.dimy;
        // ---- scanline
        uint8_t *st = a.status + h.st;
#pragma unroll 1
        for (int y = 1 + warp; y < dimy; y += kWarps)
            scan_row(h, st + (uint64_t)y * dimx, a.hoff[h.hline + y], a.hoff[h.hline + y + 1], a.hnodes + h.hnode, a.cc,
                     lane);
        // ---- column clip: points in edge order, counted, then written
        uint32_t nX = 0;
#pragma unroll 1
        for (uint32_t b = 0; b < ne && !s_full; b += NT) {
            const uint32_t e = b + tid;
            uint32_t m = 0;
            if (e < ne) m = clip_x_edge<false>(h, a.colx, a.colf, a.cert, r[e], r[e + 1], e == 0, 0, s.xc, 0u, s.xp);
            uint64_t total;
            const uint32_t at = nX + (uint32_t)small_scan<NT>(m, sums, &total);
            nX += (uint32_t)total;
            if (nX > a.cap_x) {
                if (tid == 0) s_full = 1;
            } else if (m) {
                clip_x_edge<true>(h, a.colx, a.colf, a.cert, r[e], r[e + 1], e == 0, at, s.xc, 0u, s.xp);
            }
            __syncthreads();
        }
        const uint32_t ncols = (uint32_t)h.ncols;
        if (!s_full) {
            // by column, in clip order
            uint32_t hash = 64;
            while (hash < 2 * nX) hash <<= 1;
#pragma unroll 1
            for (uint32_t i = tid; i < hash; i += NT) s.tab[i] = ~0u;
            small_bucket<NT>(
                nX, ncols, cnt, linec, sums, [&](uint32_t i) { return s.xc[i]; },
                [&](uint32_t i, uint32_t at) {
                    s.sc[at] = s.xc[i];
                    s.sp[at] = s.xp[i];
                },
                []() {});
            // duplicates: the first of a column's bit-identical points is kept,
            // found by a hash table whose slots hold the smallest index met
            auto slot_of = [&](uint32_t i, bool insert) {
                const uint64_t bits = pt_bits(s.sp[i]);
                const uint32_t c = s.sc[i];
                uint64_t k = bits ^ ((uint64_t)c << 17);
                k ^= k >> 33;
                k *= 0xff51afd7ed558ccdull;
                k ^= k >> 29;
                uint32_t t = (uint32_t)k & (hash - 1);
                for (;; t = (t + 1) & (hash - 1)) {
                    const uint32_t o = insert ? atomicCAS(&s.tab[t], ~0u, i) : *(volatile uint32_t *)&s.tab[t];
                    if (insert && o == ~0u) return t;
                    if (s.sc[o] == c && pt_bits(s.sp[o]) == bits) break;
                }
                if (insert) atomicMin(&s.tab[t], i);
                return t;
            };
            // xc keeps each point's slot from here on
#pragma unroll 1
            for (uint32_t i = tid; i < nX; i += NT) s.xc[i] = slot_of(i, true);
            __syncthreads();
            bool small = false;
#pragma unroll 1
            for (uint32_t i = tid; i < nX; i += NT) {
                const bool d = *(volatile uint32_t *)&s.tab[s.xc[i]] != i;
                s.drop[i] = d;
                small |= !d && small_pt(s.sp[i]);
            }
            if (__syncthreads_or(small)) {
                // first copies near an axis, where points closer than 1e-9 count
                // as equal: the reference's sequential rule, a column per warp
                // (the indices of the column's small points go to xc)
#pragma unroll 1
                for (uint32_t c = warp; c < ncols; c += kWarps) {
                    const uint32_t b = linec[c], e = linec[c + 1];
                    uint32_t m = 0;
#pragma unroll 1
                    for (uint32_t i0 = b; i0 < e; i0 += 32) {
                        const uint32_t i = i0 + lane;
                        const bool v = i < e && !s.drop[i] && small_pt(s.sp[i]);
                        const unsigned bm = __ballot_sync(0xffffffffu, v);
                        if (v) s.xc[b + m + __popc(bm & ((1u << lane) - 1u))] = i;
                        m += __popc(bm);
                    }
                    __syncwarp();
#pragma unroll 1
                    for (uint32_t i = 1; i < m; i++) {
                        const float2 me = s.sp[s.xc[b + i]];
                        bool eq = false;
#pragma unroll 1
                        for (uint32_t j = lane; j < i; j += 32) {
                            const uint32_t o = s.xc[b + j];
                            eq |= !s.drop[o] && pt_eq(s.sp[o], me);
                        }
                        if (__any_sync(0xffffffffu, eq) && lane == 0) s.drop[s.xc[b + i]] = 1;
                        __syncwarp();
                    }
                }
            }
            __syncthreads();
            // column polygons: kept points in order plus the closing copy of the first
#pragma unroll 1
            for (uint32_t c = warp; c < ncols; c += kWarps) {
                const uint32_t b = linec[c], e = linec[c + 1];
                uint32_t m = 0;
#pragma unroll 1
                for (uint32_t i0 = b; i0 < e; i0 += 32)
                    m += __popc(__ballot_sync(0xffffffffu, i0 + lane < e && !s.drop[i0 + lane]));
                if (lane == 0) cpst[c] = m ? m + 1 : 0u;
            }
            small_prefix<NT>(cpst, ncols, sums);
            if (cpst[ncols] > a.cap_cp && tid == 0) s_full = 1;
            __syncthreads();
        }
        if (!s_full) {
#pragma unroll 1
            for (uint32_t c = warp; c < ncols; c += kWarps) {
                const uint32_t b = linec[c], e = linec[c + 1], at = cpst[c];
                uint32_t m = 0;
                float2 f0 = make_float2(0.f, 0.f);
#pragma unroll 1
                for (uint32_t i0 = b; i0 < e; i0 += 32) {
                    const uint32_t i = i0 + lane;
                    const bool v = i < e && !s.drop[i];
                    const float2 pt = v ? s.sp[i] : f0;
                    const unsigned bm = __ballot_sync(0xffffffffu, v);
                    if (v) {
                        const uint32_t w = at + m + __popc(bm & ((1u << lane) - 1u));
                        s.cp[w] = pt;
                        s.cpc[w] = c;
                    }
                    if (m == 0 && bm) {
                        f0.x = __shfl_sync(0xffffffffu, pt.x, __ffs(bm) - 1);
                        f0.y = __shfl_sync(0xffffffffu, pt.y, __ffs(bm) - 1);
                    }
                    m += __popc(bm);
                }
                if (m && lane == 0) {
                    s.cp[at + m] = f0;
                    s.cpc[at + m] = c;
                }
            }
#pragma unroll 1
            for (uint32_t i = tid; i <= h.P; i += NT) pixc[i] = 0;
            __syncthreads();
        }
        // ---- cell clip: points in column-polygon order, counted, then written
        const uint32_t nCP = s_full ? 0u : cpst[ncols];
        uint32_t nY = 0;
#pragma unroll 1
        for (uint32_t b = 0; b < nCP && !s_full; b += NT) {
            const uint32_t j = b + tid;
            uint32_t m = 0, c = 0;
            if (j < nCP) {
                c = s.cpc[j];
                if (j + 1 < cpst[c + 1])
                    m = clip_y_edge<false>(h, a.rowy, a.rowf, a.cert, s.cp[j], s.cp[j + 1], 0, s.yr, s.yp);
            }
            uint64_t total;
            const uint32_t at = nY + (uint32_t)small_scan<NT>(m, sums, &total);
            nY += (uint32_t)total;
            if (j < nCP && j == cpst[c]) yst[c] = at;
            if (nY > a.cap_y) {
                if (tid == 0) s_full = 1;
            } else if (m) {
                clip_y_edge<true>(h, a.rowy, a.rowf, a.cert, s.cp[j], s.cp[j + 1], at, s.yr, s.yp);
            }
            __syncthreads();
        }
        if (s_full) {  // more points than the scratch holds: the pipeline takes the polygon
            if (tid == 0) {
                a.done[p] = 0;
                atomicAdd(&a.info->left, 1ull);
                atomicAdd(&a.info->crossings, 0ull - (unsigned long long)(h.n_seq > 1 ? h.n_seq - 1 : 0));
            }
            // the scanline's classes go back to the walk's border marks, as phase 1 left them
#pragma unroll 1
            for (uint32_t i = tid; i < h.P; i += NT) st[i] = st[i] == 1 ? 1 : 0;
            continue;
        }
        // by cell: a column's points stably by row (as k_cell_bucket)
        const int nrows = h.nrows;
#pragma unroll 1
        for (uint32_t c = warp; c < ncols; c += kWarps) {
            if (cpst[c + 1] == cpst[c]) continue;
            // the column's last point: the next non-empty column's first
            uint32_t e = nY;
#pragma unroll 1
            for (uint32_t d = c + 1; d < ncols; d++)
                if (cpst[d + 1] != cpst[d]) {
                    e = yst[d];
                    break;
                }
            const uint32_t b = yst[c];
#pragma unroll 1
            for (uint32_t i = b + lane; i < e; i += 32) atomicAdd(&pixc[s.yr[i] * dimx + c], 1u);
            __syncwarp();
            uint32_t base = 0;
#pragma unroll 1
            for (int r0 = 0; r0 < nrows; r0 += 32) {
                const int rr = r0 + lane;
                const uint32_t v = rr < nrows ? pixc[rr * dimx + c] : 0u;
                uint32_t incl = v;
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += u;
                }
                if (rr < nrows) pixc[rr * dimx + c] = base + incl - v;
                base += __shfl_sync(0xffffffffu, incl, 31);
            }
            __syncwarp();
            small_stable(
                0, e - b, pixc, 1, lane, [&](uint32_t i) { return s.yr[b + i] * (uint32_t)dimx + c; },
                [&](uint32_t i, uint32_t at) { s.ys[b + at] = s.yp[b + i]; });
        }
        __syncthreads();
        // ---- cell areas and classes (pixc[id] is now the end of the cell's points in its column)
#pragma unroll 1
        for (uint32_t id = tid; id < h.P; id += NT) {
            const uint32_t x = id % (uint32_t)dimx, y = id / (uint32_t)dimx;
            if (x >= ncols || y >= (uint32_t)nrows || cpst[x + 1] == cpst[x]) continue;
            const uint32_t b = y ? pixc[id - (uint32_t)dimx] : 0u;
            cell_area_class(h, id, s.ys + yst[x] + b, pixc[id] - b, st, a.areas, a.cc);
        }
        if (tid == 0) {
            atomicAdd(&a.info->clip_x, (unsigned long long)nX);
            atomicAdd(&a.info->clip_y, (unsigned long long)nY);
        }
    }
}
