// fp32-accurate projection GEMMs on exact weights, for what the 16-bit tensor-core kernels do not take: Q4_0 and Q8_0 in
// every math mode, F32 / F16 projections, K-quant rows that are no whole number of super-blocks, and the fp32 mode.
//
//   forward   Y[T, N]  = X[T, K] W[N, K]^T + bias + s low[T, R] B[R, N]      (residual += the same sum, where given)
//   backward  dX[T, K] (+)= dY[T, N] W[N, K]     + s dLow[T, R] A[K, R]^T
//
// (gemm_q4_0_batch, gemm_q8_0_batch and the *_bwd kernels of src/Glacier.Tune/Gpu/Kernels/tune_bwd.cu:131-190,335-460, and
// the rank-r terms of src/Glacier.Tune/Kernels/LoraKernels.cs:57-86,296-339.)
//
// Both operands are cut into three bf16 pieces when their tile is written to shared memory, x = x1 + x2 + x3 to 27 bits
// (each piece the rounded rest of the one before), and a product is the six bf16 MMAs x3w1, x1w3, x2w2, x2w1, x1w2, x1w1:
// what is left out is below 2^-26 of |x w|, a quarter of fp32's rounding of that product.  The MMAs of one 32-deep
// slab sum into fresh registers, and the slabs are added up in fp32: tensor cores truncate where they align addends,
// and over a whole contraction those truncations, all of one sign, would grow past fp32's own rounding.
//
// Bound: the MMA pipe (6 MMAs per 16 x 8 x 16 step) for hundreds of tokens, latency for few.  A block owns BT tokens x 64
// features; small shapes give a few dozen such tiles, so the contraction is cut over the CTAs of a cluster (up to 8),
// whose partial tiles are added in rank order through distributed shared memory: no atomics, no zero-fill, the same bits
// every run.  The rank-r term is one more slab (two above rank 32) of the same loop.
// Measured, Q8_0 896 x 4864 at 200 tokens: forward 380 -> 70 us, dX 124 -> 67 us (25 TFLOP/s; 45 at 4864 x 4992 and 1024
// tokens, where the six MMAs per product run at what mma.sync reaches on this chip, about 270 TFLOP/s) against the
// CUDA-core kernel with 64 x 64 tiles, one decoded weight per 4 multiply-adds and no split that it replaces.
#include "gt_internal.h"
#include "gt_mma.cuh"
#include "gt_ptx.cuh"
#include "gt_quant.cuh"

namespace gt {
namespace {

constexpr int BM = 64, BK = 32;            // features per block, contraction per slab
constexpr int kThreads = 256;
constexpr int kSA = (BK + 8) * 2;          // row stride of a [rows][32] 16-bit tile: 80 bytes, conflict-free for ldmatrix
constexpr int kSW = (BM + 8) * 2;          // row stride of the backward's [32 n][64 k] weight tile: 144 bytes
constexpr int kWPlane = BM * kSA;          // one plane of the weight tile (the larger of the two layouts)
static_assert(kWPlane >= BK * kSW, "weight plane holds either layout");
template <int BT>
constexpr int kStageBytes = 3 * (BT * kSA + kWPlane);
template <int BT>
constexpr int kSmemBytes = 2 * kStageBytes<BT> > BT * (BM + 4) * 4 ? 2 * kStageBytes<BT> : BT * (BM + 4) * 4;      // two stages, or the partial tile

// Eight consecutive weights of the flat element stream, still packed, and their exact fp32 values.  A run starts at a
// multiple of 8 and never crosses a block.  n_ok < 8 happens for F32 / F16 tensors only (the other types' rows are
// multiples of 32).
template <int QT>
struct Run8;
template <>
struct Run8<kTypeQ80> {
    uint16_t d, q[4];
    __device__ __forceinline__ void load(const uint8_t *w, int64_t e, int) {
        const uint8_t *b = w + (e >> 5) * kQ80BlockBytes;
        d = __ldg(reinterpret_cast<const uint16_t *>(b));
        const uint16_t *p = reinterpret_cast<const uint16_t *>(b + 2 + (e & 31));
#pragma unroll
        for (int i = 0; i < 4; i++) q[i] = __ldg(p + i);
    }
    __device__ __forceinline__ void decode(int64_t, float (&v)[8]) const {
        const float df = half_bits_to_f32(d);
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = df * (float)(int8_t)(q[i >> 1] >> (8 * (i & 1)));
    }
};
template <>
struct Run8<kTypeQ40> {
    uint16_t d, q[4];
    __device__ __forceinline__ void load(const uint8_t *w, int64_t e, int) {
        const uint8_t *b = w + (e >> 5) * kQ40BlockBytes;
        d = __ldg(reinterpret_cast<const uint16_t *>(b));
        const uint16_t *p = reinterpret_cast<const uint16_t *>(b + 2 + (e & 15));
#pragma unroll
        for (int i = 0; i < 4; i++) q[i] = __ldg(p + i);
    }
    __device__ __forceinline__ void decode(int64_t e, float (&v)[8]) const {
        const float df = half_bits_to_f32(d);
        const int sh = (e & 16) ? 4 : 0;
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = df * (float)((int)((q[i >> 1] >> (8 * (i & 1) + sh)) & 15) - 8);
    }
};
template <>
struct Run8<kTypeQ4K> {
    uint4 h;
    uint2 q;
    __device__ __forceinline__ void load(const uint8_t *w, int64_t e, int) {
        const uint8_t *b = w + (e >> 8) * kQ4KBlockBytes;
        const int c = (int)(e & 255);
        h = __ldg(reinterpret_cast<const uint4 *>(b + kQ4KHdr));
        q = __ldg(reinterpret_cast<const uint2 *>(b + (c >> 7) * 80 + ((c >> 6) & 1) * 32 + (c & 31)));
    }
    __device__ __forceinline__ void decode(int64_t e, float (&v)[8]) const {
        const int ib = (int)(e & 255) >> 5;
        int sc, m;
        q4k_scale_min_w(ib, h.y, h.z, h.w, sc, m);
        const float a = half_bits_to_f32(h.x & 0xFFFFu) * (float)sc, b = half_bits_to_f32(h.x >> 16) * (float)m;
        const uint32_t w[2] = {q.x >> ((ib & 1) * 4), q.y >> ((ib & 1) * 4)};
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = a * (float)((w[i >> 2] >> (8 * (i & 3))) & 15u) - b;
    }
};
template <>
struct Run8<kTypeQ6K> {
    uint2 l, hb;
    uint16_t d;
    int8_t sc;
    __device__ __forceinline__ void load(const uint8_t *w, int64_t e, int) {
        const uint8_t *b = w + (e >> 7) * kQ6KHalf;
        const int quad = (int)(e & 127) >> 5, ln = (int)(e & 31);
        l = __ldg(reinterpret_cast<const uint2 *>(b + 16 + (quad & 1) * 32 + ln));
        hb = __ldg(reinterpret_cast<const uint2 *>(b + 80 + ln));
        d = __ldg(reinterpret_cast<const uint16_t *>(b + 8));
        sc = __ldg(reinterpret_cast<const int8_t *>(b) + (ln >> 4) + quad * 2);
    }
    __device__ __forceinline__ void decode(int64_t e, float (&v)[8]) const {
        const int quad = ((int)(e & 127)) >> 5, ls = (quad >> 1) * 4, hs = quad * 2;
        const float a = half_bits_to_f32(d) * (float)sc;
        const uint32_t lw[2] = {l.x >> ls, l.y >> ls}, hw[2] = {hb.x >> hs, hb.y >> hs};
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int s = 8 * (i & 3);
            v[i] = a * (float)((int)(((lw[i >> 2] >> s) & 15u) | (((hw[i >> 2] >> s) & 3u) << 4)) - 32);
        }
    }
};
template <>
struct Run8<kTypeF32> {
    float f[8];
    __device__ __forceinline__ void load(const uint8_t *w, int64_t e, int n_ok) {
        const float *p = reinterpret_cast<const float *>(w) + e;
#pragma unroll
        for (int i = 0; i < 8; i++) f[i] = i < n_ok ? __ldg(p + i) : 0.f;
    }
    __device__ __forceinline__ void decode(int64_t, float (&v)[8]) const {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = f[i];
    }
};
template <>
struct Run8<kTypeF16> {
    uint16_t f[8];
    __device__ __forceinline__ void load(const uint8_t *w, int64_t e, int n_ok) {
        const uint16_t *p = reinterpret_cast<const uint16_t *>(w) + e;
#pragma unroll
        for (int i = 0; i < 8; i++) f[i] = i < n_ok ? __ldg(p + i) : (uint16_t)0;
    }
    __device__ __forceinline__ void decode(int64_t, float (&v)[8]) const {
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = half_bits_to_f32(f[i]);
    }
};

// the three bf16 pieces of a pair of values
__device__ __forceinline__ void split3(float a, float b, uint32_t (&p)[3]) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
        p[i] = *reinterpret_cast<const uint32_t *>(&v);
        a -= __uint_as_float(p[i] << 16);
        b -= __uint_as_float(p[i] & 0xFFFF0000u);
    }
}

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}

struct Args {
    const uint8_t *w;
    const float *act, *lora_act, *lora_w, *bias;
    const int *flag;
    float *out, *residual;
    float scale;
    int T, N, K, R, vec, assign;
};

// grid (feature tiles, token tiles, cluster), cluster (1, 1, S): CTA rank s of a tile's cluster takes the s-th run of slabs
template <int QT, bool BWD, int BT>
__global__ void __launch_bounds__(kThreads) k_exact_gemm(const Args p) {
    constexpr int WT = 2, WM = 8 / WT;                      // warps along tokens / features
    constexpr int MI = BT / WT / 16, NI = BM / WM / 8;      // 16-token and 8-feature MMA tiles of a warp
    constexpr int AI = BT * BK / 4 / kThreads;              // float4 of the activation tile per thread
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * BM, t0 = blockIdx.y * BT;
    const int S = gridDim.z, rank = blockIdx.z;
    const int C = BWD ? p.N : p.K, M = BWD ? p.K : p.N;
    const int n_kt = (C + BK - 1) / BK;
    pdl_wait();
    pdl_trigger();
    const bool lora = p.R > 0 && !(p.flag && *p.flag == 0);
    const int total = n_kt + (lora ? (p.R + BK - 1) / BK : 0);
    const int k_begin = total * rank / S, k_end = total * (rank + 1) / S;

    float acc[MI][NI][4];
#pragma unroll
    for (int i = 0; i < MI; i++)
#pragma unroll
        for (int j = 0; j < NI; j++) acc[i][j][0] = acc[i][j][1] = acc[i][j][2] = acc[i][j][3] = 0.f;

    // this thread's share of a slab: AI float4 of the activations, one run of eight weights
    const int a_row = tid >> 3, a_col = (tid & 7) * 4;
    const int w_row = BWD ? tid >> 3 : tid >> 2, w_run = BWD ? (tid & 7) * 8 : (tid & 3) * 8;
    float4 av[AI];
    Run8<QT> wv;
    float lw[8];
    int64_t w_e = 0;
    bool w_ok = false, is_lora = false;
    auto fetch = [&](int kt) {
        is_lora = kt >= n_kt;
        const int c0 = (is_lora ? kt - n_kt : kt) * BK;
        const float *src = is_lora ? p.lora_act : p.act;
        const int ld = is_lora ? p.R : C;
        const bool vec = (p.vec & (is_lora ? 2 : 1)) != 0;
#pragma unroll
        for (int i = 0; i < AI; i++) {
            const int t = t0 + a_row + 32 * i, c = c0 + a_col;
            av[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (t < p.T) {
                const float *q = src + (int64_t)t * ld + c;
                if (vec && c + 4 <= ld) {
                    av[i] = __ldg(reinterpret_cast<const float4 *>(q));
                } else {
                    if (c < ld) av[i].x = __ldg(q);
                    if (c + 1 < ld) av[i].y = __ldg(q + 1);
                    if (c + 2 < ld) av[i].z = __ldg(q + 2);
                    if (c + 3 < ld) av[i].w = __ldg(q + 3);
                }
            }
        }
        if (is_lora) {
            // forward: B[r, n] with r along the contraction; backward: A[k, r]
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int r = c0 + (BWD ? w_row : w_run + i), m = m0 + (BWD ? w_run + i : w_row);
                lw[i] = (r < p.R && m < M) ? p.scale * __ldg(p.lora_w + (BWD ? (int64_t)m * p.R + r : (int64_t)r * p.N + m)) : 0.f;
            }
        } else {
            const int n = BWD ? c0 + w_row : m0 + w_row, k = BWD ? m0 + w_run : c0 + w_run;
            const int n_ok = n < p.N ? min(8, p.K - k) : 0;
            w_ok = n_ok > 0;
            w_e = (int64_t)n * p.K + k;
            if (w_ok) wv.load(p.w, w_e, n_ok);
        }
    };
    auto stage = [&](int buf) {
        uint8_t *as = smem + buf * kStageBytes<BT>, *ws = as + 3 * BT * kSA;
#pragma unroll
        for (int i = 0; i < AI; i++) {
            uint32_t lo[3], hi[3];
            split3(av[i].x, av[i].y, lo);
            split3(av[i].z, av[i].w, hi);
#pragma unroll
            for (int q = 0; q < 3; q++)
                *reinterpret_cast<uint2 *>(as + q * BT * kSA + (a_row + 32 * i) * kSA + a_col * 2) = make_uint2(lo[q], hi[q]);
        }
        float v[8];
        if (is_lora) {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = lw[i];
        } else if (w_ok) {
            wv.decode(w_e, v);
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = 0.f;
        }
        uint32_t s[4][3];
#pragma unroll
        for (int i = 0; i < 4; i++) split3(v[2 * i], v[2 * i + 1], s[i]);
#pragma unroll
        for (int q = 0; q < 3; q++)
            *reinterpret_cast<uint4 *>(ws + q * kWPlane + w_row * (BWD ? kSW : kSA) + w_run * 2) = make_uint4(s[0][q], s[1][q], s[2][q], s[3][q]);
    };

    const int wt = (warp % WT) * (MI * 16), wm = (warp / WT) * (NI * 8);
    if (k_begin < k_end) {
        fetch(k_begin);
        stage(0);
    }
    __syncthreads();
    for (int kt = k_begin; kt < k_end; kt++) {
        const int buf = (kt - k_begin) & 1;
        if (kt + 1 < k_end) fetch(kt + 1);
        const uint32_t as = smem_u32(smem + buf * kStageBytes<BT>), ws = as + 3 * BT * kSA;
        float part[MI][NI][4];
#pragma unroll
        for (int i = 0; i < MI; i++)
#pragma unroll
            for (int j = 0; j < NI; j++) part[i][j][0] = part[i][j][1] = part[i][j][2] = part[i][j][3] = 0.f;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 16) {
            uint32_t a[3][MI][4], b[3][NI / 2][4];
#pragma unroll
            for (int q = 0; q < 3; q++) {
#pragma unroll
                for (int i = 0; i < MI; i++) ldsm4(a_mk(as + q * BT * kSA, kSA, wt + i * 16, kk, lane), a[q][i]);
#pragma unroll
                for (int j = 0; j < NI / 2; j++) {
                    if (BWD) ldsm4t(b_kn(ws + q * kWPlane, kSW, wm + j * 16, kk, lane), b[q][j]);
                    else ldsm4(b_nk(ws + q * kWPlane, kSA, wm + j * 16, kk, lane), b[q][j]);
                }
            }
            // smallest products first
            constexpr int pa[6] = {2, 0, 1, 1, 0, 0}, pb[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
            for (int c = 0; c < 6; c++)
#pragma unroll
                for (int i = 0; i < MI; i++)
#pragma unroll
                    for (int j = 0; j < NI; j++)
                        mma16<__nv_bfloat16>(part[i][j], a[pa[c]][i], b[pb[c]][j >> 1][(j & 1) * 2], b[pb[c]][j >> 1][(j & 1) * 2 + 1]);
        }
#pragma unroll
        for (int i = 0; i < MI; i++)
#pragma unroll
            for (int j = 0; j < NI; j++)
#pragma unroll
                for (int c = 0; c < 4; c++) acc[i][j][c] += part[i][j][c];
        if (kt + 1 < k_end) stage(buf ^ 1);      // (last read before the barrier at the end of the previous slab)
        __syncthreads();
    }

    // partial tile -> shared memory; the cluster's CTAs each sum and write BT / S token rows
    constexpr int kLd = BM + 4;
    float *tile = reinterpret_cast<float *>(smem);
#pragma unroll
    for (int i = 0; i < MI; i++)
#pragma unroll
        for (int j = 0; j < NI; j++)
#pragma unroll
            for (int h = 0; h < 2; h++)
                *reinterpret_cast<float2 *>(tile + (wt + i * 16 + (lane >> 2) + 8 * h) * kLd + wm + j * 8 + 2 * (lane & 3)) =
                    make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
    if (S > 1) cluster_sync_all();
    else __syncthreads();
    const int rows = BT / S, c4 = (tid & 15) * 4;
    for (int r = tid >> 4; r < rows; r += kThreads / 16) {
        const int tr = rank * rows + r, t = t0 + tr;
        if (t >= p.T) break;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        const uint32_t at = smem_u32(tile + tr * kLd + c4);
        for (int s = 0; s < S; s++) {
            const float4 x = S > 1 ? ld_cluster_f4(mapa_cluster(at, s)) : *reinterpret_cast<const float4 *>(tile + tr * kLd + c4);
            v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
        }
        const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int m = m0 + c4 + i;
            if (m >= M) break;
            const int64_t o = (int64_t)t * M + m;
            float x = e[i];
            if (!BWD && p.bias) x += p.bias[m];
            if (!BWD && p.residual) p.residual[o] += x;
            if (p.out) p.out[o] = (BWD && !p.assign) ? p.out[o] + x : x;
        }
    }
    if (S > 1) cluster_sync_all();      // nobody leaves while a peer still reads its tile
}

template <int QT, bool BWD, int BT>
cudaError_t launch_bt(const Args &p, int sm_count, cudaStream_t s) {
    static PerDeviceOnce configured;
    auto kern = k_exact_gemm<QT, BWD, BT>;
    cudaError_t ce = per_device_once(configured, [&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes<BT>); });
    if (ce != cudaSuccess) return ce;
    const int M = BWD ? p.K : p.N, slabs = ((BWD ? p.N : p.K) + BK - 1) / BK;
    const int64_t tiles = (int64_t)((M + BM - 1) / BM) * ((p.T + BT - 1) / BT);
    // cut the contraction while the grid stays one wave of two blocks per SM and a block keeps at least four slabs
    int S = 1;
    while (S < 8 && tiles * S * 2 <= 2 * sm_count && slabs >= 8 * S) S *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((M + BM - 1) / BM, (p.T + BT - 1) / BT, S);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes<BT>;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    unsigned na = 0;
    if (S > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = 1;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = S;
        na++;
    }
    if (pdl_enabled()) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        na++;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    return cudaLaunchKernelEx(&cfg, kern, p);
}

template <int QT, bool BWD>
cudaError_t launch_qt(const Args &p, int sm_count, cudaStream_t s) {
    // 64-token tiles reuse a decoded weight tile twice as often; 128-token ones take one block per SM (registers) and
    // measured slower at every size tried (4864 x 4992, 1024 tokens: 1159 / 1389 us)
    if (p.T <= 32) return launch_bt<QT, BWD, 32>(p, sm_count, s);
    return launch_bt<QT, BWD, 64>(p, sm_count, s);
}

}  // namespace

cudaError_t launch_exact_gemm(const ExactGemm &g, int sm_count, cudaStream_t s) {
    if (g.T <= 0 || g.N <= 0 || g.K <= 0) return cudaSuccess;
    Args p;
    p.w = g.w;
    p.act = g.act;
    p.out = g.out;
    p.residual = g.residual;
    p.bias = g.bias;
    p.T = g.T;
    p.N = g.N;
    p.K = g.K;
    p.assign = g.assign;
    p.R = (g.lora_act && g.lora_w) ? g.R : 0;
    p.lora_act = g.lora_act;
    p.lora_w = g.lora_w;
    p.scale = g.scale;
    p.flag = g.flag;
    auto aligned = [](const void *q, int ld) { return ld % 4 == 0 && (reinterpret_cast<uintptr_t>(q) & 15) == 0; };
    p.vec = (aligned(g.act, g.backward ? g.N : g.K) ? 1 : 0) | (aligned(g.lora_act, g.R) ? 2 : 0);
#define GT_EXACT(QT) return g.backward ? launch_qt<QT, true>(p, sm_count, s) : launch_qt<QT, false>(p, sm_count, s)
    switch (g.qtype) {
        case kTypeQ4K: GT_EXACT(kTypeQ4K);
        case kTypeQ6K: GT_EXACT(kTypeQ6K);
        case kTypeQ40: GT_EXACT(kTypeQ40);
        case kTypeQ80: GT_EXACT(kTypeQ80);
        case kTypeF16: GT_EXACT(kTypeF16);
        default: GT_EXACT(kTypeF32);
    }
#undef GT_EXACT
}

}  // namespace gt
