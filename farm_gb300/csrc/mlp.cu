// Learned scorer: a 520 -> 256 -> 256 -> 1 MLP (GELU; BF16 weights and
// activations on the tensor cores, FP32 accumulate), trained and run on the
// GPU with the hand-written tcgen05 GEMM of tc_gemm.cuh. It replaces the
// reference's "-a" fill-ratio confidence heuristic (query_intersect.cu:100-134):
// pairs it is sure about are decided by it, the rest go to exact refinement.
//
// Features per candidate pair (520, padded to 576 for the GEMM's K tiles):
//  * both polygons' fill classes resampled to 16 x 16 cells over the pair's
//    MBR-intersection window (cell centre -> that polygon's pixel), scaled to
//    [0, 1] and quantised to 4 bits (512 values);
//  * 8 MBR/size features: log MBR areas, window / MBR area ratios, log vertex
//    counts, log pixel counts.
//
// Training: binary cross-entropy on exact-refinement labels, Adam, mini-batches
// of 128-row multiples. Backward GEMMs run on the same kernel, which turns the
// bf16 operands of the weight gradients as it stages them (dW = dZ^T x input,
// dH = dZ x W).
#include <cuda_bf16.h>

#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"
#include "tc_gemm.cuh"

namespace farm {

constexpr int kIn = 520, kInPad = 576, kHid = 256;

struct Mlp {
    // tensor-core copies (bf16) and FP32 masters
    DevBuf W1, W2, W2T;            // bf16 [256 x 576], [256 x 256], transpose of W2
    DevBuf mW1, mW2, b1, b2, w3;   // fp32 masters; w3 holds 256 weights then b3
    DevBuf adam;                   // fp32 moments for every parameter (m, v)
    uint64_t step = 0;
    float lo = 0.02f, hi = 0.98f;  // abstain band for the learned mode
    float lambda = 0.f;            // cost-aware band: also decide when min(p, 1-p) <= lambda x cost
    bool ready = false;
    // scratch
    DevBuf X, Z1, H1, Z2, H2, dZ2, dZ1, part, gW1, gW2, gb, err;
};

static uint64_t n_params() { return (uint64_t)kHid * kInPad + kHid * kHid + kHid + kHid + kHid + 1; }

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
    float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
    float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

__device__ __forceinline__ void store16(float *d, const float *v) {
#pragma unroll
    for (int i = 0; i < 4; i++)
        reinterpret_cast<float4 *>(d)[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
}
__device__ __forceinline__ void store16(__nv_bfloat16 *d, const __nv_bfloat16 *v) {
    reinterpret_cast<uint4 *>(d)[0] = reinterpret_cast<const uint4 *>(v)[0];
    reinterpret_cast<uint4 *>(d)[1] = reinterpret_cast<const uint4 *>(v)[1];
}

// the accumulator as it is; split z of K writes its own matrix
struct EpiStoreF32 {
    float *C;
    int ldc;
    size_t split = 0;
    __device__ void operator()(int row, int col0, const float *v) const {
        float *c = C + blockIdx.z * split + (size_t)row * ldc + col0;
        if ((reinterpret_cast<uintptr_t>(c) & 15u) == 0) {
            store16(c, v);
        } else {  // the test entry takes any float boundary
#pragma unroll
            for (int i = 0; i < 16; i++) c[i] = v[i];
        }
    }
};

// z = acc + bias; keep z (fp32) and GELU(z) (bf16)
struct EpiBiasGelu {
    const float *bias;
    float *Z;
    __nv_bfloat16 *H;
    int ld;
    __device__ void operator()(int row, int col0, const float *v) const {
        float z[16];
        __align__(16) __nv_bfloat16 h[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            z[i] = v[i] + bias[col0 + i];
            h[i] = __float2bfloat16_rn(gelu(z[i]));
        }
        store16(Z + (size_t)row * ld + col0, z);
        store16(H + (size_t)row * ld + col0, h);
    }
};

// dZ = acc * GELU'(Z) (bf16), bias gradient accumulated per column: a warp's
// 32 rows are added up in registers (each step halves the columns a lane
// carries), so that an atomic stands for 32 rows. Every row is below M.
struct EpiGeluGrad {
    const float *Z;
    __nv_bfloat16 *dZ;
    float *db;
    int ld;
    __device__ void operator()(int row, int col0, const float *v) const {
        const int lane = threadIdx.x & 31;
        float d[16];
        __align__(16) __nv_bfloat16 h[16];
        const float4 *z = reinterpret_cast<const float4 *>(Z + (size_t)row * ld + col0);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float4 q = z[i];
            d[4 * i] = v[4 * i] * gelu_grad(q.x);
            d[4 * i + 1] = v[4 * i + 1] * gelu_grad(q.y);
            d[4 * i + 2] = v[4 * i + 2] * gelu_grad(q.z);
            d[4 * i + 3] = v[4 * i + 3] * gelu_grad(q.w);
        }
#pragma unroll
        for (int i = 0; i < 16; i++) h[i] = __float2bfloat16_rn(d[i]);
        store16(dZ + (size_t)row * ld + col0, h);
        int col = 0;
#pragma unroll
        for (int half = 8, o = 16; half; half >>= 1, o >>= 1) {
            const bool up = lane & o;
            col = 2 * col + (up ? 1 : 0);
#pragma unroll
            for (int i = 0; i < half; i++) {
                const float send = up ? d[i] : d[i + half], keep = up ? d[i + half] : d[i];
                d[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        d[0] += __shfl_xor_sync(0xffffffffu, d[0], 1);
        if (!(lane & 1)) atomicAdd(&db[col0 + col], d[0]);
    }
};

// grid: M / 128 x N / BN x splits of K, k_per elements each (a multiple of 64)
template <int BN, bool kT, typename Epi>
__global__ void __launch_bounds__(tc::kThreads) k_gemm(const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *B,
                                                       int ldb, int M, int N, int K, int k_per, int *err, Epi epi) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const int kb = (int)blockIdx.z * k_per;
    tc::gemm_tile<BN, kT>(A, lda, B, ldb, M, N, kb, min(K, kb + k_per), blockIdx.x * tc::kBM, blockIdx.y * BN, smem,
                          err, epi);
}

template <int BN, bool kT, typename Epi>
static int launch_gemm(const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *B, int ldb, int M, int N, int K,
                       int splits, int k_per, int *err, Epi epi, cudaStream_t st) {
    constexpr int smem = tc::smem_bytes<BN>();
    FARM_CUDA(cudaFuncSetAttribute(k_gemm<BN, kT, Epi>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    dim3 grid((M + tc::kBM - 1) / tc::kBM, (N + BN - 1) / BN, splits);
    k_gemm<BN, kT, Epi><<<grid, tc::kThreads, smem, st>>>(A, lda, B, ldb, M, N, K, k_per, err, epi);
    FARM_CUDA(cudaGetLastError());
    return FARM_OK;
}

// ------------------------------------------------------------ features --

// The reference cell of sample c (one axis): the pixel of lo + (c + 0.5)
// (hi - lo) / 16, the grid cell centre, in a raster starting at m[0] (m[2] its
// end) of `dim` pixels; -1 when the centre lies outside the raster's box.
__device__ __noinline__ int sample_cell_fp64(double w0, double w1, int c, double m0, double m2, double step, int dim) {
    const double v = w0 + (c + 0.5) * (w1 - w0) / 16.0;
    if (v < m0 || v > m2) return -1;
    int x = double_to_int((v - m0) / step);
    x = x < 0 ? 0 : x;
    return x > dim - 1 ? dim - 1 : x;
}

// log or ratio feature of a pair (the FP64 expressions, decided on bf16 by
// pair_features where FP32 leaves the rounding open)
__device__ __noinline__ float size_feature_fp64(int k, double as, double at, double aw, uint32_t snv, uint32_t tnv,
                                                uint32_t sP, uint32_t tP) {
    switch (k) {
        case 0: return (float)(log(as + 1e-12) / 10.0);
        case 1: return (float)(log(at + 1e-12) / 10.0);
        case 2: return (float)(aw / (as + 1e-30));
        case 3: return (float)(aw / (at + 1e-30));
        case 4: return (float)(log((double)snv) / 10.0);
        case 5: return (float)(log((double)tnv) / 10.0);
        case 6: return (float)(log((double)sP + 1.0) / 10.0);
        default: return (float)(log((double)tP + 1.0) / 10.0);
    }
}

// Fill class s (of cc) as a feature: the fill ratio quantised to 4 bits (w = 4).
__device__ __forceinline__ __nv_bfloat16 class_feature(int s, int cc) {
    const float r = (float)s / (float)(cc - 1);
    return __float2bfloat16_rn(rintf(r * 15.f) / 15.f);
}

// The features of one pair, by a warp: put(k, value) for k in [0, kInPad).
//
// A cell's pixel is an FP64 quotient truncated, and a size feature an FP64
// logarithm rounded to bf16; FP64 issues at 2 lanes per clock per SM, so both
// are taken in FP32 with an error bound and in FP64 only where the truncation
// or the rounding is not certain. A grid row's and a grid column's pixels are
// computed once per pair (lane l: column l & 15 and row l >> 1 of either
// polygon) instead of once per cell: 64 instead of 1,024 quotients a pair.
// lut: class_feature of every class. 65,536 pairs: 3,040 us with an FP64
// quotient per cell and FP64 logarithms.
template <typename Put>
__device__ __forceinline__ void pair_features(const StoreView &sv, const PolyHdr &S, const PolyHdr &T,
                                              const __nv_bfloat16 *lut, int cc, int lane, Put put) {
    const unsigned full = 0xffffffffu;
    // lanes 0-15: the 16 columns, 16-31: the 16 rows
    const int ax = lane >> 4, c = lane & 15;
    const double s0 = S.mbr[ax], s1 = S.mbr[2 + ax], t0 = T.mbr[ax], t1 = T.mbr[2 + ax];
    const double w0 = fmax(s0, t0);
    double w1 = fmin(s1, t1);
    if (w1 < w0) w1 = w0;
    const double width = w1 - w0;
    const float wf = (float)width, big = (float)fmax(fabs(w0), fabs(w1));
    // boxes that do not overlap, or by less than the coordinates resolve:
    // cells can lie outside, every one goes through FP64
    const bool thin = !(wf > 1e-12f * big);
    int cell[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const PolyHdr &H = k ? T : S;
        const double m0 = k ? t0 : s0, m2 = k ? t1 : s1, step = ax ? H.step_y : H.step_x;
        const int dim = ax ? H.dimy : H.dimx;
        const float st = (float)step;
        const float a = __fdiv_rn((float)(w0 - m0), st), b = __fdiv_rn(wf, st);
        const float q = __fmaf_rn((c + 0.5f) * 0.0625f, b, a);
        const float margin = 1e-6f * (a + b + 1.f) + 4e-15f * __fdiv_rn(big, st) + 2e-8f;
        const float fl = floorf(q);
        if (thin || !(q < 4e6f) || q - fl < margin || fl + 1.f - q < margin)
            cell[k] = sample_cell_fp64(w0, w1, c, m0, m2, step, dim);
        else
            cell[k] = min(max((int)fl, 0), dim - 1);
    }
    const uint8_t *sst = sv.status + S.st, *tst = sv.status + T.st;
    const int sx = __shfl_sync(full, cell[0], c), tx = __shfl_sync(full, cell[1], c);
#pragma unroll
    for (int t = 0; t < 8; t++) {
        const int gy = 2 * t + ax;
        const int sy = __shfl_sync(full, cell[0], 16 + gy), ty = __shfl_sync(full, cell[1], 16 + gy);
        int vs = 0, vt = 0;
        if (!S.err && sx >= 0 && sy >= 0) vs = sst[(uint32_t)(sy * S.dimx + sx)];
        if (!T.err && tx >= 0 && ty >= 0) vt = tst[(uint32_t)(ty * T.dimx + tx)];
        put(32 * t + lane, lut[vs]);
        put(256 + 32 * t + lane, lut[vt]);
    }
    // size features: lane k < 8 (k even: source, odd: target), then the padding
    const double wy = __shfl_sync(full, width, 16), wx = __shfl_sync(full, width, 0);
    if (lane < 8) {
        const double as = (S.mbr[2] - S.mbr[0]) * (S.mbr[3] - S.mbr[1]);
        const double at = (T.mbr[2] - T.mbr[0]) * (T.mbr[3] - T.mbr[1]);
        const double aw = wx * wy;
        const bool odd = lane & 1;
        const float area = (float)(odd ? at : as);
        const float n = (float)((lane >> 1) == 2 ? (odd ? T.nv : S.nv) : (odd ? T.P : S.P) + 1u);
        const float v = (lane >> 1) == 1 ? __fdiv_rn((float)aw, area)
                                         : __fmul_rn(logf((lane >> 1) == 0 ? __fadd_rn(area, 1e-12f) : n), 0.1f);
        const float e = __fadd_rn(__fmul_rn(1e-6f, fabsf(v)), 1e-7f);
        const __nv_bfloat16 lo = __float2bfloat16_rn(v - e), hi = __float2bfloat16_rn(v + e);
        const bool sure = area > 1e-20f && __bfloat16_as_ushort(lo) == __bfloat16_as_ushort(hi);
        put(512 + lane, sure ? lo : __float2bfloat16_rn(size_feature_fp64(lane, as, at, aw, S.nv, T.nv, S.P, T.P)));
    }
    for (int k = kIn + lane; k < kInPad; k += 32) put(k, __float2bfloat16_rn(0.f));
}

// one warp per pair; rows >= n are zero padding
__global__ void __launch_bounds__(256) k_features(const StoreView sv, const uint32_t *__restrict__ pairs, uint64_t n,
                                                  uint64_t rows, uint64_t tgt_base, __nv_bfloat16 *__restrict__ X) {
    __shared__ __nv_bfloat16 lut[256];
    const int lane = threadIdx.x & 31;
    const int cc = sv.category_count;
    lut[threadIdx.x] = class_feature((int)threadIdx.x, cc);
    __syncthreads();
    uint64_t w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t r = w; r < rows; r += nw) {
        __nv_bfloat16 *x = X + r * kInPad;
        if (r >= n) {
            for (int k = lane; k < kInPad; k += 32) x[k] = __float2bfloat16_rn(0.f);
            continue;
        }
        pair_features(sv, sv.hdr[pairs[2 * r]], sv.hdr[tgt_base + pairs[2 * r + 1]], lut, cc, lane,
                      [&](int k, __nv_bfloat16 v) { x[k] = v; });
    }
}

// --------------------------------------------------- the fused scorer --

constexpr int kScoreThreads = 512;
constexpr uint32_t kXBytes = tc::kBM * kInPad * 2;          // the features of 128 pairs
constexpr uint32_t kWBytes = kHid * tc::kBK * 2;            // a 64-wide slice of a weight matrix
constexpr uint32_t kScoreSmem = kXBytes + 2 * kWBytes + 4 * (3 * kHid + 1) + 16 + 512 + 64;
constexpr int kScoreChunks = kInPad / tc::kBK + kHid / tc::kBK;  // slices of W1, then of W2

// Probabilities of n pairs in one kernel: a CTA takes 128 pairs at a time,
// builds their features in shared memory in the tensor core's layout, runs
// both hidden layers there (weights streamed from L2 in 64-wide slices, two in
// flight) and keeps every activation on chip. Before, features, both layers'
// pre-activations and activations and the logits went through memory in four
// kernels per 65,536 pairs. The arithmetic is theirs, operation for operation:
// the same products in the same order, the same roundings, the logit summed
// over the lanes as k_logit sums it. What bounds it is instruction issue (the
// features, and the two GELUs of 256 x 128 values a tile); one CTA of 16 warps
// per SM, as the features and two weight slices fill its shared memory.
// 200,003 pairs: 11.9 ms before, 0.74 ms so.
__global__ void __launch_bounds__(kScoreThreads, 1)
    k_score(const StoreView sv, const uint32_t *__restrict__ pairs, uint64_t n, uint64_t tgt_base,
            const __nv_bfloat16 *__restrict__ W1, const __nv_bfloat16 *__restrict__ W2, const float *__restrict__ b1,
            const float *__restrict__ b2, const float *__restrict__ w3, float *__restrict__ prob, int *err) {
    extern __shared__ __align__(1024) unsigned char smem[];
    constexpr uint32_t kSboX = kInPad * 16, kSboH = kHid * 16;  // bytes per 8 rows
    unsigned char *X = smem;                              // features; then layer 1's activations,
    unsigned char *H2 = smem + tc::kBM * kHid * 2;        // and layer 2's behind them
    unsigned char *Wst = smem + kXBytes;
    float *sb1 = reinterpret_cast<float *>(Wst + 2 * kWBytes), *sb2 = sb1 + kHid, *sw3 = sb2 + kHid;
    __nv_bfloat16 *lut = reinterpret_cast<__nv_bfloat16 *>(sw3 + kHid + 4);
    uint64_t *bar = reinterpret_cast<uint64_t *>((reinterpret_cast<uintptr_t>(lut + 256) + 7) & ~(uintptr_t)7);
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 2);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cc = sv.category_count;
    if (tid == 0) {
        tc::mbar_init(&bar[0], 1);
        tc::mbar_init(&bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int k = tid; k < kHid; k += kScoreThreads) {
        sb1[k] = b1[k];
        sb2[k] = b2[k];
        sw3[k] = w3[k];
        lut[k] = class_feature(k, cc);
    }
    if (tid == 0) sw3[kHid] = w3[kHid];
    if (warp == 0) tc::tmem_alloc(tslot, 256);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *tslot;
    const uint32_t idesc = tc::make_idesc(tc::kBM, kHid);
    uint32_t phase[2] = {0, 0};
    bool ok = true;
    // slice c of a tile's weights (W1 then W2) into stage s; a tile has an odd
    // number of slices, so a slice's stage alternates from tile to tile
    uint32_t run = 0;  // slices multiplied so far
    auto load_slice = [&](int c, uint32_t s) {
        const bool first = c < kInPad / tc::kBK;
        const __nv_bfloat16 *W = first ? W1 : W2;
        const int ld = first ? kInPad : kHid, k0 = (first ? c : c - kInPad / tc::kBK) * tc::kBK;
        const uint32_t dst = tc::smem_addr(Wst + s * kWBytes);
        for (int v = tid; v < kHid * 8; v += kScoreThreads) {
            const int r = v >> 3, kc = v & 7;
            tc::cp_async16(dst + tc::tile_off((uint32_t)r, (uint32_t)(kc * 8)), W + (size_t)r * ld + k0 + kc * 8);
        }
    };
    // one slice: its MMAs, then (once they have read it) the slice two on
    auto step = [&](const unsigned char *A, uint32_t sbo, int kslice, int kk_n, int next) {
        tc::cp_async_wait<1>();
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        const uint32_t s = run++ & 1;
        if (tid == 0 && ok) {
            for (int kk = 0; kk < kk_n; kk++) {
                const uint64_t ad = tc::make_desc_sbo(tc::smem_addr(A) + (kslice * 8 + kk * 2) * tc::kLBO, sbo);
                const uint64_t bd = tc::make_desc(tc::smem_addr(Wst + s * kWBytes) + kk * 2 * tc::kLBO);
                tc::mma_bf16(tmem, ad, bd, idesc, (kslice > 0 || kk > 0) ? 1u : 0u);
            }
            tc::mma_commit(&bar[s]);
        }
        ok = ok && tc::mbar_wait(&bar[s], phase[s]);
        phase[s] ^= 1;
        if (next >= 0) load_slice(next, s);
        tc::cp_async_commit();  // one group per step, empty ones too
    };
    // z = accumulator + bias, GELU(z) in bf16 into dst (row pitch kSboH per 8 rows)
    auto activate = [&](const float *bias, unsigned char *dst) {
        const int row = (warp & 3) * 32 + lane;
        for (int c = (warp >> 2) * 64; c < (warp >> 2) * 64 + 64; c += 16) {
            float v[16];
            tc::tmem_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c, v);
            __nv_bfloat16 h[16];
#pragma unroll
            for (int i = 0; i < 16; i++) h[i] = __float2bfloat16_rn(gelu(v[i] + bias[c + i]));
            unsigned char *d = dst + (row >> 3) * kSboH + (c >> 3) * tc::kLBO + (row & 7) * 16;
            *reinterpret_cast<uint4 *>(d) = *reinterpret_cast<const uint4 *>(h);
            *reinterpret_cast<uint4 *>(d + tc::kLBO) = *reinterpret_cast<const uint4 *>(h + 8);
        }
    };
    const uint64_t tiles = (n + tc::kBM - 1) / tc::kBM;
    if (blockIdx.x < tiles) {
        load_slice(0, 0);
        tc::cp_async_commit();
        load_slice(1, 1);
        tc::cp_async_commit();
    }
    for (uint64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const bool last = tile + gridDim.x >= tiles;
        const uint64_t r0 = tile * tc::kBM;
        for (int r = warp; r < tc::kBM; r += kScoreThreads / 32) {
            unsigned char *xr = X + (r >> 3) * kSboX + (r & 7) * 16;
            auto put = [&](int k, __nv_bfloat16 v) {
                *reinterpret_cast<__nv_bfloat16 *>(xr + (k >> 3) * tc::kLBO + (k & 7) * 2) = v;
            };
            if (r0 + r < n) {
                const uint2 pq = load_pair(pairs, r0 + r);
                pair_features(sv, sv.hdr[pq.x], sv.hdr[tgt_base + pq.y], lut, cc, lane, put);
            } else {
                for (int k = lane; k < kInPad; k += 32) put(k, __float2bfloat16_rn(0.f));
            }
        }
        // layer 1: features 520 and up are zero padding and add nothing
        for (int c = 0; c < kInPad / tc::kBK; c++) {
            const int left = (kIn - c * tc::kBK + 15) / 16;
            step(X, kSboX, c, left < 4 ? left : 4, c + 2);
        }
        tc::fence_after_sync();
        activate(sb1, X);
        // layer 2
        for (int c = 0; c < kHid / tc::kBK; c++) {
            const int next = kInPad / tc::kBK + c + 2;
            step(X, kSboH, c, 4, next < kScoreChunks ? next : (last ? -1 : next - kScoreChunks));
        }
        tc::fence_after_sync();
        activate(sb2, H2);
        tc::fence_before_sync();
        __syncthreads();
        for (int r = warp; r < tc::kBM && r0 + r < n; r += kScoreThreads / 32) {
            const unsigned char *h = H2 + (r >> 3) * kSboH + (r & 7) * 16;
            float z = 0;
            for (int j = lane; j < kHid; j += 32)
                z += __bfloat162float(*reinterpret_cast<const __nv_bfloat16 *>(h + (j >> 3) * tc::kLBO + (j & 7) * 2)) *
                     sw3[j];
            for (int o = 16; o; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
            if (lane == 0) prob[r0 + r] = 1.f / (1.f + expf(-(z + sw3[kHid])));
        }
        __syncthreads();  // the next tile's features overwrite the activations
    }
    tc::cp_async_wait<0>();
    if (!ok && lane == 0) atomicExch(err, 1);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 256);
}

// ------------------------------------------------- elementwise kernels --

// The head, forward and backward, a warp per row: the logit H2[r] . w3 + b3,
// BCE with logits (dlogit = (sigmoid - y) / n, loss sum), dZ2 = dlogit * w3 *
// GELU'(Z2) in bf16, and the gradients of w3, b3 and b2, which each lane adds
// up for its 8 columns over the warp's rows, each block over its warps, so
// that an atomic stands for a block's rows. Rows >= n (padding) get zero
// gradient. It replaced three kernels that wrote the logits out and added
// every row's every column by atomics.
__global__ void __launch_bounds__(256) k_head(const __nv_bfloat16 *__restrict__ H2, const float *__restrict__ Z2,
                                              const float *__restrict__ w3, const uint8_t *__restrict__ y, uint64_t n,
                                              uint64_t rows, __nv_bfloat16 *__restrict__ dZ2, float *__restrict__ db2,
                                              float *__restrict__ dw3, float *__restrict__ db3,
                                              float *__restrict__ loss) {
    __shared__ float acc[2 * kHid];
    const int lane = threadIdx.x & 31;
    acc[threadIdx.x] = 0.f;
    acc[kHid + threadIdx.x] = 0.f;
    __syncthreads();
    float w[8], g3[8], g2[8], my_loss = 0, my_b3 = 0;
#pragma unroll
    for (int t = 0; t < 8; t++) {
        w[t] = w3[lane + 32 * t];
        g3[t] = g2[t] = 0.f;
    }
    const float b3 = w3[kHid];
    const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5;
    for (uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += nw) {
        float h[8], s = 0;
#pragma unroll
        for (int t = 0; t < 8; t++) {
            h[t] = __bfloat162float(H2[r * kHid + lane + 32 * t]);
            s += h[t] * w[t];
        }
        for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        float d = 0;
        if (r < n) {
            const float z = s + b3, t = (float)y[r];
            const float p = 1.f / (1.f + expf(-z));
            d = (p - t) / (float)n;
            my_loss += (fmaxf(z, 0.f) - z * t + log1pf(expf(-fabsf(z)))) / (float)n;
            my_b3 += d;
        }
#pragma unroll
        for (int t = 0; t < 8; t++) {
            const int j = lane + 32 * t;
            const float e = r < n ? d * w[t] * gelu_grad(Z2[r * kHid + j]) : 0.f;
            dZ2[r * kHid + j] = __float2bfloat16_rn(e);
            if (d != 0) g3[t] += d * h[t];  // padding may hold anything, infinities and NaN too
            g2[t] += e;
        }
    }
#pragma unroll
    for (int t = 0; t < 8; t++) {
        atomicAdd(&acc[lane + 32 * t], g3[t]);
        atomicAdd(&acc[kHid + lane + 32 * t], g2[t]);
    }
    if (lane == 0 && my_loss != 0) atomicAdd(loss, my_loss);
    if (lane == 0 && my_b3 != 0) atomicAdd(db3, my_b3);
    __syncthreads();
    atomicAdd(&dw3[threadIdx.x], acc[threadIdx.x]);
    atomicAdd(&db2[threadIdx.x], acc[kHid + threadIdx.x]);
}

// The splits' partial weight gradients added up in order: n1 elements of s1
// partials, then n2 of s2.
__global__ void k_sum_splits(const float *__restrict__ p1, uint64_t n1, int s1, float *__restrict__ g1,
                             const float *__restrict__ p2, uint64_t n2, int s2, float *__restrict__ g2) {
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n1 + n2;
         k += (uint64_t)gridDim.x * blockDim.x) {
        const bool a = k < n1;
        const float *p = a ? p1 + k : p2 + (k - n1);
        const uint64_t step = a ? n1 : n2;
        float s = 0;
        for (int z = 0; z < (a ? s1 : s2); z++) s += p[z * step];
        (a ? g1 : g2)[a ? k : k - n1] = s;
    }
}

// dst[c][r] = src[r][c] for a [R x C] bf16 matrix, 32 x 32 tiles via shared memory
__global__ void k_transpose(const __nv_bfloat16 *__restrict__ src, uint64_t R, uint64_t Cc,
                            __nv_bfloat16 *__restrict__ dst) {
    __shared__ __nv_bfloat16 tile[32][33];
    uint64_t bx = blockIdx.x * 32ull, by = blockIdx.y * 32ull;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        uint64_t r = by + i, c = bx + threadIdx.x;
        tile[i][threadIdx.x] = (r < R && c < Cc) ? src[r * Cc + c] : __float2bfloat16_rn(0.f);
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        uint64_t c = bx + i, r = by + threadIdx.x;
        if (c < Cc && r < R) dst[c * R + r] = tile[threadIdx.x][i];
    }
}

__global__ void k_to_bf16(const float *__restrict__ a, uint64_t n, __nv_bfloat16 *__restrict__ b) {
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (uint64_t)gridDim.x * blockDim.x)
        b[k] = __float2bfloat16_rn(a[k]);
}

// Adam (beta1 0.9, beta2 0.999); grad scaled by gscale
__global__ void k_adam(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, uint64_t n, float lr, float bc1, float bc2) {
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (uint64_t)gridDim.x * blockDim.x) {
        float gk = g[k];
        float mk = 0.9f * m[k] + 0.1f * gk, vk = 0.999f * v[k] + 0.001f * gk * gk;
        m[k] = mk;
        v[k] = vk;
        p[k] -= lr * (mk / bc1) / (sqrtf(vk / bc2) + 1e-8f);
    }
}

// deterministic small-scale uniform init in [-a, a]
__global__ void k_init(float *__restrict__ p, uint64_t n, float a, uint64_t seed) {
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t z = seed * 0x9E3779B97F4A7C15ull + k;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        p[k] = a * (2.f * ((float)(z >> 40) / 16777216.f) - 1.f);
    }
}

__global__ void k_gather_rows(const __nv_bfloat16 *__restrict__ X, const uint32_t *__restrict__ idx, uint64_t n,
                              uint64_t rows, const uint8_t *__restrict__ yin, __nv_bfloat16 *__restrict__ out,
                              uint8_t *__restrict__ yout) {
    for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < rows * kInPad;
         k += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t r = k / kInPad, c = k % kInPad;
        out[k] = r < n ? X[(uint64_t)idx[r] * kInPad + c] : __float2bfloat16_rn(0.f);
        if (c == 0) yout[r] = r < n ? yin[idx[r]] : 0;
    }
}

static unsigned gbm(uint64_t n) {
    uint64_t g = (n + 255) / 256;
    uint64_t cap = 64ull * sm_count();
    if (g > cap) g = cap;
    return (unsigned)(g ? g : 1);
}

void mlp_free(void *p) {
    Mlp *m = static_cast<Mlp *>(p);
    if (!m) return;
    DevBuf *b[] = {&m->W1, &m->W2, &m->W2T, &m->mW1, &m->mW2, &m->b1, &m->b2, &m->w3, &m->adam, &m->X, &m->Z1,
                   &m->H1, &m->Z2, &m->H2, &m->dZ2, &m->dZ1, &m->part, &m->gW1, &m->gW2, &m->gb, &m->err};
    for (DevBuf *x : b) x->release();
    delete m;
}

float mlp_band(farm_store *s, int which) {
    Mlp *m = static_cast<Mlp *>(s->mlp);
    return m ? (which == 2 ? m->lambda : (which ? m->hi : m->lo)) : 0.f;
}

static Mlp *mlp_of(farm_store *s) {
    if (!s->mlp) s->mlp = new Mlp();
    return static_cast<Mlp *>(s->mlp);
}

static int mlp_alloc(Mlp *m) {
    FARM_TRY(m->W1.ensure(2ull * kHid * kInPad));
    FARM_TRY(m->W2.ensure(2ull * kHid * kHid));
    FARM_TRY(m->W2T.ensure(2ull * kHid * kHid));
    FARM_TRY(m->mW1.ensure(4ull * kHid * kInPad));
    FARM_TRY(m->mW2.ensure(4ull * kHid * kHid));
    FARM_TRY(m->b1.ensure(4 * kHid));
    FARM_TRY(m->b2.ensure(4 * kHid));
    FARM_TRY(m->w3.ensure(4 * (kHid + 1)));
    FARM_TRY(m->adam.ensure(8 * n_params()));
    FARM_TRY(m->err.ensure(64));
    return FARM_OK;
}

// refresh the bf16 copies from the masters
static int mlp_sync_bf16(Mlp *m, cudaStream_t st) {
    k_to_bf16<<<gbm(kHid * kInPad), 256, 0, st>>>(m->mW1.as<float>(), (uint64_t)kHid * kInPad,
                                                  m->W1.as<__nv_bfloat16>());
    k_to_bf16<<<gbm(kHid * kHid), 256, 0, st>>>(m->mW2.as<float>(), (uint64_t)kHid * kHid, m->W2.as<__nv_bfloat16>());
    dim3 tb(32, 8), tg(kHid / 32, kHid / 32);
    k_transpose<<<tg, tb, 0, st>>>(m->W2.as<__nv_bfloat16>(), kHid, kHid, m->W2T.as<__nv_bfloat16>());
    FARM_CUDA(cudaGetLastError());
    return FARM_OK;
}

// forward over `rows` (multiple of 128) feature rows in X, up to the second
// layer's activations (k_head goes on from there). Tiles are 128 x 64: a batch
// of 4,096 rows fills 128 SMs, 32 of them with 128 x 256.
static int mlp_forward(Mlp *m, const __nv_bfloat16 *X, uint64_t rows, cudaStream_t st) {
    FARM_TRY(m->Z1.ensure(4 * rows * kHid));
    FARM_TRY(m->H1.ensure(2 * rows * kHid));
    FARM_TRY(m->Z2.ensure(4 * rows * kHid));
    FARM_TRY(m->H2.ensure(2 * rows * kHid));
    int *err = m->err.as<int>();
    EpiBiasGelu e1{m->b1.as<float>(), m->Z1.as<float>(), m->H1.as<__nv_bfloat16>(), kHid};
    FARM_TRY((launch_gemm<64, false>(X, kInPad, m->W1.as<__nv_bfloat16>(), kInPad, (int)rows, kHid, kInPad, 1, kInPad,
                                     err, e1, st)));
    EpiBiasGelu e2{m->b2.as<float>(), m->Z2.as<float>(), m->H2.as<__nv_bfloat16>(), kHid};
    FARM_TRY((launch_gemm<64, false>(m->H1.as<__nv_bfloat16>(), kHid, m->W2.as<__nv_bfloat16>(), kHid, (int)rows, kHid,
                                     kHid, 1, kHid, err, e2, st)));
    return FARM_OK;
}

// rows per split of a weight gradient's product over the rows: `base` (a
// multiple of 64), more when that makes over 64 splits
static int split_rows(uint64_t rows, int base) {
    const uint64_t least = ((rows + 63) / 64 + 63) & ~63ull;
    return (int)(least > (uint64_t)base ? least : (uint64_t)base);
}

// gradients into m->gW1, m->gW2, m->gb (b1 | b2 | w3 | b3), loss into *loss
// (device). The weight gradients are products over the rows with 256 x 256 and
// 256 x 576 results, 4 and 9 tiles: the rows are split so that the chip is
// filled, and the partial products added up in order. Against 64 bits over 4,096
// rows of the same bf16 operands a product of 512 or 256 rows a split is off by
// 1.1e-7 or 5e-8 of its largest element (rms), one accumulator by 1.0e-6.
static int mlp_backward(Mlp *m, const __nv_bfloat16 *X, const uint8_t *y, uint64_t n, uint64_t rows, float *dloss,
                        cudaStream_t st) {
    const int k1 = split_rows(rows, 512), k2 = split_rows(rows, 256);
    const int s1 = (int)((rows + k1 - 1) / k1), s2 = (int)((rows + k2 - 1) / k2);
    const uint64_t n1 = (uint64_t)kHid * kInPad, n2 = (uint64_t)kHid * kHid;
    FARM_TRY(m->dZ2.ensure(2 * rows * kHid));
    FARM_TRY(m->dZ1.ensure(2 * rows * kHid));
    FARM_TRY(m->part.ensure(4 * (n1 * s1 + n2 * s2)));
    FARM_TRY(m->gW1.ensure(4 * n1));
    FARM_TRY(m->gW2.ensure(4 * n2));
    FARM_TRY(m->gb.ensure(4ull * (3 * kHid + 1) + 64));
    float *gb = m->gb.as<float>();
    float *db1 = gb, *db2 = gb + kHid, *dw3 = gb + 2 * kHid, *db3 = gb + 3 * kHid;
    FARM_CUDA(cudaMemsetAsync(gb, 0, 4ull * (3 * kHid + 1), st));
    int *err = m->err.as<int>();
    const __nv_bfloat16 *H1 = m->H1.as<__nv_bfloat16>(), *dZ1 = m->dZ1.as<__nv_bfloat16>(),
                        *dZ2 = m->dZ2.as<__nv_bfloat16>();
    const uint64_t hb = (rows + 31) / 32;  // 4 rows a warp
    k_head<<<(unsigned)(hb < 2048 ? hb : 2048), 256, 0, st>>>(m->H2.as<__nv_bfloat16>(), m->Z2.as<float>(),
                                                              m->w3.as<float>(), y, n, rows,
                                                              m->dZ2.as<__nv_bfloat16>(), db2, dw3, db3, dloss);
    // dW2 = dZ2^T x H1, both given by rows
    float *p1 = m->part.as<float>(), *p2 = p1 + n1 * s1;
    FARM_TRY((launch_gemm<64, true>(dZ2, kHid, H1, kHid, kHid, kHid, (int)rows, s2, k2, err,
                                    EpiStoreF32{p2, kHid, n2}, st)));
    // dH1 = dZ2 x W2 -> dZ1 = dH1 * GELU'(Z1) : A = dZ2 [rows x 256], B = W2^T [256 x 256]
    EpiGeluGrad eg{m->Z1.as<float>(), m->dZ1.as<__nv_bfloat16>(), db1, kHid};
    FARM_TRY((launch_gemm<64, false>(dZ2, kHid, m->W2T.as<__nv_bfloat16>(), kHid, (int)rows, kHid, kHid, 1, kHid, err,
                                     eg, st)));
    // dW1 = dZ1^T x X
    FARM_TRY((launch_gemm<64, true>(dZ1, kHid, X, kInPad, kHid, kInPad, (int)rows, s1, k1, err,
                                    EpiStoreF32{p1, kInPad, n1}, st)));
    k_sum_splits<<<gbm(n1 + n2), 256, 0, st>>>(p1, n1, s1, m->gW1.as<float>(), p2, n2, s2, m->gW2.as<float>());
    FARM_CUDA(cudaGetLastError());
    return FARM_OK;
}

static int mlp_adam(Mlp *m, float lr, cudaStream_t st) {
    m->step++;
    float bc1 = 1.f - powf(0.9f, (float)m->step), bc2 = 1.f - powf(0.999f, (float)m->step);
    float *am = m->adam.as<float>(), *av = am + n_params();
    uint64_t o = 0;
    auto upd = [&](float *p, const float *g, uint64_t n) {
        k_adam<<<gbm(n), 256, 0, st>>>(p, g, am + o, av + o, n, lr, bc1, bc2);
        o += n;
    };
    const float *gb = m->gb.as<float>();
    upd(m->mW1.as<float>(), m->gW1.as<float>(), (uint64_t)kHid * kInPad);
    upd(m->mW2.as<float>(), m->gW2.as<float>(), (uint64_t)kHid * kHid);
    upd(m->b1.as<float>(), gb, kHid);
    upd(m->b2.as<float>(), gb + kHid, kHid);
    upd(m->w3.as<float>(), gb + 2 * kHid, kHid + 1);  // w3 and b3
    FARM_CUDA(cudaGetLastError());
    return FARM_OK;
}

static int check_err(Mlp *m, cudaStream_t st) {
    int h = 0;
    FARM_CUDA(cudaMemcpyAsync(&h, m->err.p, 4, cudaMemcpyDeviceToHost, st));
    FARM_CUDA(cudaStreamSynchronize(st));
    if (h) {
        set_error("tcgen05 GEMM: an mbarrier wait timed out");
        return FARM_ETIMEOUT;
    }
    return FARM_OK;
}

static uint64_t pad128(uint64_t n) { return (n + 127) & ~127ull; }

}  // namespace farm

using namespace farm;

extern "C" {

/* Test hook of the tcgen05 GEMM (see farm_gpu.h). */
int farm_tc_gemm_test(const void *A, const void *B, float *C, int M, int N, int K, int BN) {
    if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0 || M % 16 || N % 16 || K % 64) {
        set_error("farm_tc_gemm_test: bad shape");
        return FARM_EINVAL;
    }
    int *err = nullptr;
    FARM_CUDA(cudaMalloc(&err, 4));
    FARM_CUDA(cudaMemset(err, 0, 4));
    const __nv_bfloat16 *a = static_cast<const __nv_bfloat16 *>(A), *b = static_cast<const __nv_bfloat16 *>(B);
    EpiStoreF32 epi{C, N};
    int rc;
    if (BN == 64)
        rc = launch_gemm<64, false>(a, K, b, K, M, N, K, 1, K, err, epi, 0);
    else if (BN == 128)
        rc = launch_gemm<128, false>(a, K, b, K, M, N, K, 1, K, err, epi, 0);
    else
        rc = launch_gemm<256, false>(a, K, b, K, M, N, K, 1, K, err, epi, 0);
    int herr = 0;
    if (rc == FARM_OK) {
        cudaError_t e = cudaMemcpy(&herr, err, 4, cudaMemcpyDeviceToHost);
        if (e != cudaSuccess) rc = cuda_fail(e, "farm_tc_gemm_test");
    }
    cudaFree(err);
    if (rc == FARM_OK && herr) {
        set_error("farm_tc_gemm_test: an mbarrier wait timed out");
        return FARM_ETIMEOUT;
    }
    return rc;
}

int farm_mlp_init(farm_store *s, uint64_t seed) {
    if (!s) return FARM_EINVAL;
    Mlp *m = mlp_of(s);
    FARM_TRY(mlp_alloc(m));
    cudaStream_t st = s->stream;
    float a1 = sqrtf(6.f / (kIn + kHid)), a2 = sqrtf(6.f / (2 * kHid)), a3 = sqrtf(6.f / (kHid + 1));
    k_init<<<gbm(kHid * kInPad), 256, 0, st>>>(m->mW1.as<float>(), (uint64_t)kHid * kInPad, a1, seed * 4 + 1);
    k_init<<<gbm(kHid * kHid), 256, 0, st>>>(m->mW2.as<float>(), (uint64_t)kHid * kHid, a2, seed * 4 + 2);
    k_init<<<gbm(kHid), 256, 0, st>>>(m->w3.as<float>(), kHid, a3, seed * 4 + 3);
    FARM_CUDA(cudaMemsetAsync(m->w3.as<float>() + kHid, 0, 4, st));
    FARM_CUDA(cudaMemsetAsync(m->b1.p, 0, 4 * kHid, st));
    FARM_CUDA(cudaMemsetAsync(m->b2.p, 0, 4 * kHid, st));
    FARM_CUDA(cudaMemsetAsync(m->adam.p, 0, 8 * n_params(), st));
    m->step = 0;
    FARM_TRY(mlp_sync_bf16(m, st));
    FARM_CUDA(cudaStreamSynchronize(st));
    m->ready = true;
    s->launches += 6;
    return FARM_OK;
}

/* Features of n candidate pairs into X (device, bf16 [n_pad x 576]). */
int farm_mlp_features(farm_store *s, const uint32_t *d_pairs, uint64_t n, void *d_X, uint64_t rows) {
    if (!s || !s->rasterized || rows < n) return FARM_EINVAL;
    FARM_TRY(check_pairs(s, d_pairs, n, FARM_MEM_DEVICE, false, "farm_mlp_features"));
    k_features<<<gbm(32 * rows), 256, 0, s->stream>>>(s->view(), d_pairs, n, rows, s->n_side[0],
                                                      static_cast<__nv_bfloat16 *>(d_X));
    FARM_CUDA(cudaGetLastError());
    FARM_CUDA(cudaStreamSynchronize(s->stream));
    s->launches++;
    return FARM_OK;
}

/* One forward + backward on given features (device bf16 [rows x 576], rows a
 * multiple of 128) and labels (device u8, first n rows): loss and gradients in
 * the layout of farm_mlp_get (W1 | W2 | b1 | b2 | w3 | b3), no update. */
int farm_mlp_grad(farm_store *s, const void *d_X, const uint8_t *d_y, uint64_t n, uint64_t rows, float *h_loss,
                  float *h_grad) {
    if (!s || !s->mlp || rows % 128 || rows < n) return FARM_EINVAL;
    Mlp *m = mlp_of(s);
    cudaStream_t st = s->stream;
    // the GEMMs read rows 16 bytes at a time
    const __nv_bfloat16 *X = static_cast<const __nv_bfloat16 *>(d_X);
    if (reinterpret_cast<uintptr_t>(d_X) & 15u) {
        FARM_TRY(m->X.ensure(2 * rows * kInPad));
        FARM_CUDA(cudaMemcpyAsync(m->X.p, d_X, 2 * rows * kInPad, cudaMemcpyDeviceToDevice, st));
        X = m->X.as<__nv_bfloat16>();
    }
    FARM_CUDA(cudaMemsetAsync(m->err.p, 0, 4, st));
    float *dloss;
    FARM_TRY(s->d_counters.ensure(256));
    dloss = s->d_counters.as<float>();
    FARM_CUDA(cudaMemsetAsync(dloss, 0, 4, st));
    FARM_TRY(mlp_forward(m, X, rows, st));
    FARM_TRY(mlp_backward(m, X, d_y, n, rows, dloss, st));
    FARM_TRY(check_err(m, st));
    if (h_loss) FARM_CUDA(cudaMemcpy(h_loss, dloss, 4, cudaMemcpyDeviceToHost));
    if (h_grad) {
        float *o = h_grad;
        FARM_CUDA(cudaMemcpy(o, m->gW1.p, 4ull * kHid * kInPad, cudaMemcpyDeviceToHost));
        o += (uint64_t)kHid * kInPad;
        FARM_CUDA(cudaMemcpy(o, m->gW2.p, 4ull * kHid * kHid, cudaMemcpyDeviceToHost));
        o += (uint64_t)kHid * kHid;
        FARM_CUDA(cudaMemcpy(o, m->gb.p, 4ull * (3 * kHid + 1), cudaMemcpyDeviceToHost));
    }
    return FARM_OK;
}

uint64_t farm_mlp_param_count(void) { return n_params(); }

/* Decision band of the learned mode: probability >= hi decides 1, <= lo
 * decides 0, anything between goes to exact refinement. */
int farm_mlp_set_band(farm_store *s, float lo, float hi) {
    if (!s || !(lo <= hi) || !isfinite(lo) || !isfinite(hi)) {
        set_error("farm_mlp_set_band: need finite lo <= hi");
        return FARM_EINVAL;
    }
    Mlp *m = mlp_of(s);
    m->lo = lo;
    m->hi = hi;
    return FARM_OK;
}

int farm_mlp_set_band_cost(farm_store *s, float lambda) {
    if (!s || !(lambda >= 0.f) || !isfinite(lambda)) {
        set_error("farm_mlp_set_band_cost: need a finite lambda >= 0");
        return FARM_EINVAL;
    }
    mlp_of(s)->lambda = lambda;
    return FARM_OK;
}

/* Copy the FP32 master parameters out / in (W1 [256 x 576] | W2 [256 x 256] |
 * b1 | b2 | w3 | b3). */
int farm_mlp_get(farm_store *s, float *out) {
    if (!s || !s->mlp || !out) return FARM_EINVAL;
    Mlp *m = mlp_of(s);
    FARM_CUDA(cudaStreamSynchronize(s->stream));
    float *o = out;
    FARM_CUDA(cudaMemcpy(o, m->mW1.p, 4ull * kHid * kInPad, cudaMemcpyDeviceToHost));
    o += (uint64_t)kHid * kInPad;
    FARM_CUDA(cudaMemcpy(o, m->mW2.p, 4ull * kHid * kHid, cudaMemcpyDeviceToHost));
    o += (uint64_t)kHid * kHid;
    FARM_CUDA(cudaMemcpy(o, m->b1.p, 4 * kHid, cudaMemcpyDeviceToHost));
    o += kHid;
    FARM_CUDA(cudaMemcpy(o, m->b2.p, 4 * kHid, cudaMemcpyDeviceToHost));
    o += kHid;
    FARM_CUDA(cudaMemcpy(o, m->w3.p, 4 * (kHid + 1), cudaMemcpyDeviceToHost));
    return FARM_OK;
}

int farm_mlp_set(farm_store *s, const float *in) {
    if (!s || !in) return FARM_EINVAL;
    Mlp *m = mlp_of(s);
    FARM_TRY(mlp_alloc(m));
    const float *o = in;
    FARM_CUDA(cudaMemcpy(m->mW1.p, o, 4ull * kHid * kInPad, cudaMemcpyHostToDevice));
    o += (uint64_t)kHid * kInPad;
    FARM_CUDA(cudaMemcpy(m->mW2.p, o, 4ull * kHid * kHid, cudaMemcpyHostToDevice));
    o += (uint64_t)kHid * kHid;
    FARM_CUDA(cudaMemcpy(m->b1.p, o, 4 * kHid, cudaMemcpyHostToDevice));
    o += kHid;
    FARM_CUDA(cudaMemcpy(m->b2.p, o, 4 * kHid, cudaMemcpyHostToDevice));
    o += kHid;
    FARM_CUDA(cudaMemcpy(m->w3.p, o, 4 * (kHid + 1), cudaMemcpyHostToDevice));
    FARM_CUDA(cudaMemset(m->adam.p, 0, 8 * n_params()));
    m->step = 0;
    FARM_TRY(mlp_sync_bf16(m, s->stream));
    FARM_CUDA(cudaStreamSynchronize(s->stream));
    m->ready = true;
    return FARM_OK;
}

/* Train on n candidate pairs (device pairs, device u8 labels from exact
 * refinement): epochs x shuffled mini-batches of `batch` rows (multiple of
 * 128), Adam with learning rate lr. Returns the last epoch's mean loss. */
int farm_mlp_train(farm_store *s, const uint32_t *d_pairs, const uint8_t *d_labels, uint64_t n, int epochs,
                   int batch, float lr, uint64_t seed, float *last_loss) {
    if (!s || !s->rasterized || !d_pairs || !d_labels || n == 0 || batch <= 0 || batch % 128) return FARM_EINVAL;
    FARM_TRY(check_pairs(s, d_pairs, n, FARM_MEM_DEVICE, false, "farm_mlp_train"));
    Mlp *m = mlp_of(s);
    if (!m->ready) FARM_TRY(farm_mlp_init(s, seed));
    cudaStream_t st = s->stream;
    const uint64_t rows_all = pad128(n);
    DevBuf &Xall = s->s[Q_SCR0], &perm = s->s[Q_SCR1], &yb = s->s[Q_SCR2];
    FARM_TRY(Xall.ensure(2 * rows_all * kInPad));
    k_features<<<gbm(32 * rows_all), 256, 0, st>>>(s->view(), d_pairs, n, rows_all, s->n_side[0],
                                                   Xall.as<__nv_bfloat16>());
    FARM_TRY(m->X.ensure(2ull * batch * kInPad));
    FARM_TRY(yb.ensure((uint64_t)batch + 64));
    FARM_TRY(perm.ensure(4 * n));
    FARM_TRY(s->d_counters.ensure(256));
    float *dloss = s->d_counters.as<float>();
    FARM_CUDA(cudaMemsetAsync(m->err.p, 0, 4, st));
    std::vector<uint32_t> hp(n);
    uint64_t rng = seed * 0x9E3779B97F4A7C15ull + 12345;
    float loss = 0;
    for (int ep = 0; ep < epochs; ep++) {
        for (uint64_t i = 0; i < n; i++) hp[i] = (uint32_t)i;
        for (uint64_t i = n - 1; i > 0; i--) {  // Fisher-Yates with a splitmix stream
            rng += 0x9E3779B97F4A7C15ull;
            uint64_t z = rng;
            z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
            z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
            z ^= z >> 31;
            uint64_t j = z % (i + 1);
            uint32_t t = hp[i];
            hp[i] = hp[j];
            hp[j] = t;
        }
        FARM_CUDA(cudaMemcpyAsync(perm.p, hp.data(), 4 * n, cudaMemcpyHostToDevice, st));
        FARM_CUDA(cudaMemsetAsync(dloss, 0, 4, st));
        uint64_t nb = 0;
        for (uint64_t b0 = 0; b0 < n; b0 += (uint64_t)batch, nb++) {
            uint64_t nn = n - b0 < (uint64_t)batch ? n - b0 : (uint64_t)batch;
            uint64_t rows = pad128(nn);
            k_gather_rows<<<gbm(rows * kInPad), 256, 0, st>>>(Xall.as<__nv_bfloat16>(), perm.as<uint32_t>() + b0, nn,
                                                              rows, d_labels, m->X.as<__nv_bfloat16>(),
                                                              yb.as<uint8_t>());
            FARM_TRY(mlp_forward(m, m->X.as<__nv_bfloat16>(), rows, st));
            FARM_TRY(mlp_backward(m, m->X.as<__nv_bfloat16>(), yb.as<uint8_t>(), nn, rows, dloss, st));
            FARM_TRY(mlp_adam(m, lr, st));
            FARM_TRY(mlp_sync_bf16(m, st));
        }
        FARM_CUDA(cudaMemcpyAsync(&loss, dloss, 4, cudaMemcpyDeviceToHost, st));
        FARM_CUDA(cudaStreamSynchronize(st));
        loss /= (float)(nb ? nb : 1);
    }
    FARM_TRY(check_err(m, st));
    if (last_loss) *last_loss = loss;
    return FARM_OK;
}

/* Probabilities for n pairs (device pairs -> device fp32 out). */
int farm_mlp_predict(farm_store *s, const uint32_t *d_pairs, uint64_t n, float *d_prob) {
    if (!s || !s->mlp || !s->rasterized) return FARM_EINVAL;
    Mlp *m = mlp_of(s);
    if (!m->ready) {
        set_error("no trained scorer in this store");
        return FARM_EINVAL;
    }
    FARM_TRY(check_pairs(s, d_pairs, n, FARM_MEM_DEVICE, false, "farm_mlp_predict"));
    cudaStream_t st = s->stream;
    FARM_CUDA(cudaMemsetAsync(m->err.p, 0, 4, st));
    if (n) {
        FARM_CUDA(cudaFuncSetAttribute(k_score, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScoreSmem));
        const uint64_t tiles = (n + tc::kBM - 1) / tc::kBM, most = (uint64_t)sm_count();
        k_score<<<(unsigned)(tiles < most ? tiles : most), kScoreThreads, kScoreSmem, st>>>(
            s->view(), d_pairs, n, s->n_side[0], m->W1.as<__nv_bfloat16>(), m->W2.as<__nv_bfloat16>(),
            m->b1.as<float>(), m->b2.as<float>(), m->w3.as<float>(), d_prob, m->err.as<int>());
        FARM_CUDA(cudaGetLastError());
        s->launches++;
    }
    FARM_TRY(check_err(m, st));
    return FARM_OK;
}

}  // extern "C"
