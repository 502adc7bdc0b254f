// Causal multi-head attention with grouped KV heads, forward and backward, without the [heads, T, T] buffers.
//
// Replaces tune_attn_causal_gqa_fwd / tune_attn_causal_gqa_bwd_dq_ds / tune_attn_causal_gqa_bwd_dk_dv
// (src/Glacier.Tune/Gpu/Kernels/tune_bwd.cu:527-717, launched from src/Glacier.Tune/Gpu/GpuLoraEngine.Forward.cs:433-513
// and GpuLoraEngine.Backward.cs:354-459) and their CPU statement CausalAttentionKernel.Forward / Backward
// (src/Glacier.Tune/Kernels/CausalAttentionKernel.cs:17-213).  The reference stores the softmax rows (attnProbs
// [heads_q, T, T]) in the forward and a dS buffer of the same size in the backward; here the forward keeps one
// log-sum-exp per (head, query) and the backward recomputes the probabilities tile by tile.
//
//   scores = q k^T / sqrt(head_dim), key j visible to query i iff j <= i; head h reads KV head h / (heads_q / heads_kv)
//   out = softmax(scores) v
//   dP = dO v^T;  dS = P * (dP - rowsum(dO * out)) / sqrt(head_dim);  dq = dS k;  dk = dS^T q;  dv = P^T dO
//
// Layouts as the reference: q, out, dO, dq [T, heads_q, head_dim]; k, v, dk, dv [T, heads_kv, head_dim], fp32 at the boundary.
// The kernels read 16-bit copies of q, k, v and dO, rounded once (bf16 in the bf16 math mode, fp16 in the validation modes) by
// k_attn_operands (which also rotates q and k inside a training step and scales q by log2(e) / sqrt(head_dim): scores are kept
// in the base-2 domain) and k_attn_delta; products run on warp-level m16n8k16 MMAs with fp32 accumulation and fp32 softmax
// statistics.  A warp owns 16 rows of a tile and keeps its probabilities in registers: the accumulator fragment of one product
// is the operand fragment of the next, so a tile costs two barriers (the double-buffered tiles that cp.async fills) and no
// shared-memory round trip.  Bound: the mma.sync pipe, 576 TFLOP/s at 1.9 GHz (m16n8k16: 2 clocks per SM).
//   k_attn_fwd      grid (heads_q, query tiles, longest first): online softmax over the key tiles at or left of the diagonal
//   k_attn_delta    rowsum(dO * out) per (head, query), and the 16-bit copy of dO
//   k_attn_bwd      grid (2 * heads_q, tiles, longest first): even blocks: dq of one query tile, summed over its key tiles in
//                   registers; odd blocks: dk, dv of one key tile for ONE query head, summed over the query tiles in
//                   registers, written to a per-query-head workspace
//   k_attn_reduce_kv sums the query heads of each KV group (fixed order: results do not change from run to run)
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cmath>

#include "gt_engine_priv.h"
#include "gt_mma.cuh"
#include "gt_ptx.cuh"

using gt::launch_k;
using gt::pdl_trigger;
using gt::pdl_wait;

using namespace gt;

namespace {

constexpr int D = 128;              // head_dim served
constexpr int BK = 64;              // key tile; query tile of the backward
constexpr int SD = (D + 8) * 2;     // smem row stride in bytes of a [rows][128] 16-bit tile (272: conflict-free ldmatrix)
constexpr int kTile = BK * SD;

template <typename T16>
__device__ __forceinline__ uint32_t pk(float lo, float hi);
template <>
__device__ __forceinline__ uint32_t pk<__nv_bfloat16>(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
}
template <>
__device__ __forceinline__ uint32_t pk<__half>(float lo, float hi) {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
}

__device__ __forceinline__ void cp16(uint32_t dst, const void *src, bool live) {      // 16 bytes, zeros where not live
    const int n = live ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const void *src, bool live) {
    const int n = live ? 4 : 0;
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// rows t0 .. t0 + ROWS - 1 of one head of a 16-bit [T, heads, 128] tensor -> shared memory, rows at or beyond T as zeros
template <int ROWS, int NT>
__device__ __forceinline__ void fetch_tile(const uint16_t *__restrict__ src, int64_t ld, int col0, int t0, int T, uint32_t dst, int tid) {
#pragma unroll
    for (int i = 0; i < ROWS * 16 / NT; i++) {
        const int idx = tid + i * NT, r = idx >> 4, c = idx & 15, t = t0 + r;
        const bool live = t < T;
        cp16(dst + r * SD + c * 16, src + (int64_t)(live ? t : 0) * ld + col0 + c * 8, live);
    }
}

constexpr float kLog2e = 1.4426950408889634f;
// 2^x on the special-function unit (2 ulp; 2^-inf = 0): the probabilities are rounded to 16 bits right after
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// ------------------------------------------------------------------------------------------------ 16-bit operands
// One block per position: q16 = scale * q, k16 = k (both rotated first when freq_base > 0: RoPE as k_rope in gt_glue.cu, same
// fp32 order), v16 = v.
template <typename T16>
__global__ void __launch_bounds__(256) k_attn_operands(const float *__restrict__ q, const float *__restrict__ k, const float *__restrict__ v,
                                                       uint16_t *__restrict__ q16, uint16_t *__restrict__ k16, uint16_t *__restrict__ v16, int HQ, int HK,
                                                       float freq_base, float qscale) {
    __shared__ __align__(16) float cs[D / 2], sn[D / 2];
    pdl_wait();
    pdl_trigger();
    const int pos = blockIdx.x, tid = threadIdx.x;
    if (tid < D / 2) {
        float c = 1.f, sv = 0.f;
        if (freq_base > 0.f) {
            const float base_freq = 1.0f / powf(freq_base, (float)(2 * tid) / (float)D);
            sincosf((float)pos * base_freq * 1.0f, &sv, &c);
        }
        cs[tid] = c;
        sn[tid] = sv;
    }
    __syncthreads();
    for (int it = tid; it < (HQ + HK) * (D / 8); it += 256) {
        const int h = it >> 4, i = (it & 15) * 4;
        const bool is_q = h < HQ;
        const int64_t off = is_q ? ((int64_t)pos * HQ + h) * D + i : ((int64_t)pos * HK + (h - HQ)) * D + i;
        const float *src = (is_q ? q : k) + off;
        const float4 a = *reinterpret_cast<const float4 *>(src), b = *reinterpret_cast<const float4 *>(src + D / 2);
        const float4 c = *reinterpret_cast<const float4 *>(cs + i), z = *reinterpret_cast<const float4 *>(sn + i);
        const float sc = is_q ? qscale : 1.f;
        uint16_t *dst = (is_q ? q16 : k16) + off;
        *reinterpret_cast<uint2 *>(dst) = make_uint2(pk<T16>((a.x * c.x - b.x * z.x) * sc, (a.y * c.y - b.y * z.y) * sc),
                                                     pk<T16>((a.z * c.z - b.z * z.z) * sc, (a.w * c.w - b.w * z.w) * sc));
        *reinterpret_cast<uint2 *>(dst + D / 2) = make_uint2(pk<T16>((a.x * z.x + b.x * c.x) * sc, (a.y * z.y + b.y * c.y) * sc),
                                                             pk<T16>((a.z * z.z + b.z * c.z) * sc, (a.w * z.w + b.w * c.w) * sc));
    }
    for (int it = tid; it < HK * (D / 4); it += 256) {
        const int64_t off = (int64_t)pos * HK * D + it * 4;
        const float4 a = *reinterpret_cast<const float4 *>(v + off);
        *reinterpret_cast<uint2 *>(v16 + off) = make_uint2(pk<T16>(a.x, a.y), pk<T16>(a.z, a.w));
    }
}

// ------------------------------------------------------------------------------------------------ forward
// WQ warps along the query tile (16 rows each) x WK groups that take every WK-th key tile with buffers of their own and join
// their softmax states at the end.  8 x 1 reuses a key tile for 128 queries; 4 x 2 halves the length of the chain of key tiles,
// which is what short sequences wait for.
template <int WQ, int WK>
constexpr int kFwdSmem = 16 * WQ * SD + WK * 4 * kTile;
template <typename T16, int WQ, int WK>
__global__ void __launch_bounds__(32 * WQ * WK, 1) k_attn_fwd(const uint16_t *__restrict__ q, const uint16_t *__restrict__ k, const uint16_t *__restrict__ v,
                                                              float *__restrict__ out, uint16_t *__restrict__ out16, float *__restrict__ lse2, int T,
                                                              int HQ, int HK) {
    constexpr int BQ = 16 * WQ, NG = 32 * WQ;      // queries per block, threads per group
    pdl_wait();
    pdl_trigger();
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int grp = tid / NG, gt = tid - grp * NG, wq = gt >> 5;
    const int h = blockIdx.x, kh = h / (HQ / HK), it = (int)gridDim.y - 1 - (int)blockIdx.y;
    const int q0 = it * BQ, last = min(q0 + BQ, T) - 1;
    const int64_t ldq = (int64_t)HQ * D, ldk = (int64_t)HK * D;
    const uint32_t qs = smem_u32(smem), kv = qs + BQ * SD + grp * 4 * kTile;      // K0, V0, K1, V1
    auto group_sync = [&] {
        if (WK == 1) __syncthreads();
        else asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(NG) : "memory");
    };
    auto fetch = [&](int jt, int buf) {
        if (jt * BK <= last) {
            fetch_tile<BK, NG>(k, ldk, kh * D, jt * BK, T, kv + buf * 2 * kTile, gt);
            fetch_tile<BK, NG>(v, ldk, kh * D, jt * BK, T, kv + (buf * 2 + 1) * kTile, gt);
        }
        cp_commit();
    };
    fetch_tile<BQ, 32 * WQ * WK>(q, ldq, h * D, q0, T, qs, tid);
    fetch(grp, 0);
    cp_wait<0>();
    __syncthreads();
    uint32_t qf[D / 16][4];
#pragma unroll
    for (int kk = 0; kk < D / 16; kk++) ldsm4(a_mk(qs, SD, wq * 16, kk * 16, lane), qf[kk]);
    float o[D / 8][4];
#pragma unroll
    for (int n = 0; n < D / 8; n++) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
    const int row[2] = {q0 + wq * 16 + g, q0 + wq * 16 + g + 8};
    const int wlast = q0 + wq * 16 + 15;      // the warp's last query
    for (int jt = grp, buf = 0; jt * BK <= last; jt += WK, buf ^= 1) {
        const int k0 = jt * BK;
        fetch(jt + WK, buf ^ 1);
        cp_wait<1>();
        group_sync();      // tile jt is in place for every warp of the group
        if (k0 <= wlast) {
            const uint32_t ks = kv + buf * 2 * kTile, vs = ks + kTile;
            float s[BK / 8][4];
#pragma unroll
            for (int n = 0; n < BK / 8; n++) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
            for (int kk = 0; kk < D / 16; kk++) {
#pragma unroll
                for (int n = 0; n < BK / 8; n += 2) {
                    uint32_t b[4];
                    ldsm4(b_nk(ks, SD, n * 8, kk * 16, lane), b);
                    mma16<T16>(s[n], qf[kk], b[0], b[1]);
                    mma16<T16>(s[n + 1], qf[kk], b[2], b[3]);
                }
            }
            // causal mask where the tile reaches past the warp's first query (keys beyond T lie past every query in range)
            if (k0 + BK - 1 > q0 + wq * 16) {
#pragma unroll
                for (int n = 0; n < BK / 8; n++) {
#pragma unroll
                    for (int c = 0; c < 4; c++)
                        if (k0 + n * 8 + 2 * t4 + (c & 1) > row[c >> 1]) s[n][c] = -INFINITY;
                }
            }
            float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int n = 0; n < BK / 8; n++) {
                mx[0] = fmaxf(mx[0], fmaxf(s[n][0], s[n][1]));
                mx[1] = fmaxf(mx[1], fmaxf(s[n][2], s[n][3]));
            }
            float corr[2];
#pragma unroll
            for (int r = 0; r < 2; r++) {
                mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 1));
                mx[r] = fmaxf(mx[r], __shfl_xor_sync(0xffffffffu, mx[r], 2));
                // a finite floor keeps (-inf) - (-inf) out of the exponent (a row all of whose keys in this tile are masked)
                const float mn = fmaxf(fmaxf(m[r], mx[r]), -3.0e38f);
                corr[r] = ex2(m[r] - mn);
                m[r] = mn;
            }
            float ps[2] = {0.f, 0.f};
            uint32_t pf[BK / 16][4];
#pragma unroll
            for (int n = 0; n < BK / 8; n++) {
                const float p0 = ex2(s[n][0] - m[0]), p1 = ex2(s[n][1] - m[0]);
                const float p2 = ex2(s[n][2] - m[1]), p3 = ex2(s[n][3] - m[1]);
                ps[0] += p0 + p1;
                ps[1] += p2 + p3;
                pf[n >> 1][(n & 1) * 2] = pk<T16>(p0, p1);
                pf[n >> 1][(n & 1) * 2 + 1] = pk<T16>(p2, p3);
            }
#pragma unroll
            for (int r = 0; r < 2; r++) l[r] = l[r] * corr[r] + ps[r];
            // the running maxima move in the first tiles and then rarely: rescale the accumulator only when one did
            if (__any_sync(0xffffffffu, corr[0] != 1.f || corr[1] != 1.f)) {
#pragma unroll
                for (int n = 0; n < D / 8; n++) {
                    o[n][0] *= corr[0];
                    o[n][1] *= corr[0];
                    o[n][2] *= corr[1];
                    o[n][3] *= corr[1];
                }
            }
#pragma unroll
            for (int kk = 0; kk < BK / 16; kk++) {
#pragma unroll
                for (int n = 0; n < D / 8; n += 2) {
                    uint32_t b[4];
                    ldsm4t(b_kn(vs, SD, n * 8, kk * 16, lane), b);
                    mma16<T16>(o[n], pf[kk], b[0], b[1]);
                    mma16<T16>(o[n + 1], pf[kk], b[2], b[3]);
                }
            }
        }
        group_sync();      // the tile's buffer is free
    }
    cp_wait<0>();
#pragma unroll
    for (int r = 0; r < 2; r++) {
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 1);
        l[r] += __shfl_xor_sync(0xffffffffu, l[r], 2);
    }
    if (WK > 1) {
        // groups 1.. hand their state over in shared memory (their own tile buffers), group 0 joins them in group order
        constexpr int kLdO = D + 4;
        float *st = reinterpret_cast<float *>(smem + BQ * SD + grp * 4 * kTile);      // [BQ][kLdO] sums, then m, l [BQ] each
        if (grp > 0) {
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int lr = wq * 16 + g + 8 * r;
#pragma unroll
                for (int n = 0; n < D / 8; n++) *reinterpret_cast<float2 *>(st + lr * kLdO + n * 8 + 2 * t4) = make_float2(o[n][2 * r], o[n][2 * r + 1]);
                if (t4 == 0) {
                    st[BQ * kLdO + lr] = m[r];
                    st[BQ * kLdO + BQ + lr] = l[r];
                }
            }
        }
        __syncthreads();
        if (grp > 0) return;
#pragma unroll
        for (int x = 1; x < WK; x++) {
            const float *sx = reinterpret_cast<const float *>(smem + BQ * SD + x * 4 * kTile);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const int lr = wq * 16 + g + 8 * r;
                const float mo = sx[BQ * kLdO + lr], mn = fmaxf(fmaxf(m[r], mo), -3.0e38f);
                const float c0 = ex2(m[r] - mn), c1 = ex2(mo - mn);
                m[r] = mn;
                l[r] = l[r] * c0 + sx[BQ * kLdO + BQ + lr] * c1;
#pragma unroll
                for (int n = 0; n < D / 8; n++) {
                    const float2 w = *reinterpret_cast<const float2 *>(sx + lr * kLdO + n * 8 + 2 * t4);
                    o[n][2 * r] = o[n][2 * r] * c0 + w.x * c1;
                    o[n][2 * r + 1] = o[n][2 * r + 1] * c0 + w.y * c1;
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        if (row[r] >= T) continue;
        const float inv = l[r] > 0.f ? 1.f / l[r] : 0.f;
        float *dst = out + (int64_t)row[r] * ldq + h * D;
#pragma unroll
        for (int n = 0; n < D / 8; n++) *reinterpret_cast<float2 *>(dst + n * 8 + 2 * t4) = make_float2(o[n][2 * r] * inv, o[n][2 * r + 1] * inv);
        if (out16) {      // the operand of the output projection: no cast pass has to read the fp32 copy back
            uint16_t *d16 = out16 + (int64_t)row[r] * ldq + h * D;
#pragma unroll
            for (int n = 0; n < D / 8; n++) *reinterpret_cast<uint32_t *>(d16 + n * 8 + 2 * t4) = pack2<T16>(o[n][2 * r] * inv, o[n][2 * r + 1] * inv);
        }
        if (t4 == 0) lse2[(int64_t)h * T + row[r]] = m[r] + log2f(l[r]);
    }
}

// delta[h, t] = sum_d dO[t, h, d] * out[t, h, d], and dO16 = dO rounded; one warp per (t, h)
template <typename T16>
__global__ void k_attn_delta(const float *__restrict__ d_out, const float *__restrict__ out, float *__restrict__ delta, uint16_t *__restrict__ do16, int T,
                             int HQ) {
    pdl_wait();
    pdl_trigger();
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= T * HQ) return;
    const int t = w / HQ, h = w % HQ;
    const int64_t off = ((int64_t)t * HQ + h) * D + lane * 4;
    const float4 a = __ldg(reinterpret_cast<const float4 *>(d_out + off));
    const float4 b = __ldg(reinterpret_cast<const float4 *>(out + off));
    *reinterpret_cast<uint2 *>(do16 + off) = make_uint2(pk<T16>(a.x, a.y), pk<T16>(a.z, a.w));
    float s = a.x * b.x + a.y * b.y + a.z * b.z + a.w * b.w;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) delta[(int64_t)h * T + t] = s;
}

// ------------------------------------------------------------------------------------------------ backward
// Both kinds of block: WK groups of 4 warps that take every WK-th tile with buffers of their own and add up at the end; one
// group per block and two blocks per SM for long sequences, two groups and one block where the blocks are few and the chain of
// tiles is what counts.  P = exp2(S2 - lse2), dS = P (dP - delta) / sqrt(D).
constexpr int kGrp = 128;      // threads of a group
constexpr int kLdAcc = D + 4;
template <int WK>
constexpr int kBwdSmem = 2 * kTile + WK * (4 * kTile + 4 * BK * 4);
static_assert(4 * kTile >= 2 * BK * kLdAcc * 4, "a group's sums fit its tile buffers");
template <int WK>
__device__ __forceinline__ void bwd_group_sync(int grp) {
    if (WK == 1) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + grp), "n"(kGrp) : "memory");
}
// acc of group 0 += acc of the others, handed over in shared memory at st[group] (fixed order); false for groups that are done
template <int WK, int NA>
__device__ __forceinline__ bool bwd_join(float (&acc)[NA][D / 8][4], float *const (&st)[WK], int grp, int m0, int g, int t4) {
    if (WK == 1) return true;
    if (grp > 0) {
#pragma unroll
        for (int a = 0; a < NA; a++)
#pragma unroll
            for (int n = 0; n < D / 8; n++)
#pragma unroll
                for (int r = 0; r < 2; r++)
                    *reinterpret_cast<float2 *>(st[grp] + (a * BK + m0 + g + 8 * r) * kLdAcc + n * 8 + 2 * t4) = make_float2(acc[a][n][2 * r], acc[a][n][2 * r + 1]);
    }
    __syncthreads();
    if (grp > 0) return false;
#pragma unroll
    for (int x = 1; x < WK; x++)
#pragma unroll
        for (int a = 0; a < NA; a++)
#pragma unroll
            for (int n = 0; n < D / 8; n++)
#pragma unroll
                for (int r = 0; r < 2; r++) {
                    const float2 w = *reinterpret_cast<const float2 *>(st[x] + (a * BK + m0 + g + 8 * r) * kLdAcc + n * 8 + 2 * t4);
                    acc[a][n][2 * r] += w.x;
                    acc[a][n][2 * r + 1] += w.y;
                }
    return true;
}

// dq[query tile] = sum over key tiles j <= i of dS K; a warp owns 16 queries
template <typename T16, int WK>
__device__ __forceinline__ void attn_bwd_dq_block(const uint16_t *__restrict__ d_out, const uint16_t *__restrict__ q, const uint16_t *__restrict__ k,
                                                  const uint16_t *__restrict__ v, const float *__restrict__ lse2, const float *__restrict__ delta,
                                                  float *__restrict__ dq, int T, int HQ, int HK, int h, int it) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x, grp = tid / kGrp, gt = tid - grp * kGrp, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int kh = h / (HQ / HK), q0 = it * BK, m0 = (gt >> 5) * 16;
    const int64_t ldq = (int64_t)HQ * D, ldk = (int64_t)HK * D;
    const uint32_t qs = smem_u32(smem), dos = qs + kTile, kv = qs + (2 + 4 * grp) * kTile;      // K0, V0, K1, V1
    auto fetch = [&](int jt, int buf) {
        if (jt <= it) {
            fetch_tile<BK, kGrp>(k, ldk, kh * D, jt * BK, T, kv + buf * 2 * kTile, gt);
            fetch_tile<BK, kGrp>(v, ldk, kh * D, jt * BK, T, kv + (buf * 2 + 1) * kTile, gt);
        }
        cp_commit();
    };
    fetch_tile<BK, WK * kGrp>(q, ldq, h * D, q0, T, qs, tid);
    fetch_tile<BK, WK * kGrp>(d_out, ldq, h * D, q0, T, dos, tid);
    fetch(grp, 0);
    float sum[1][D / 8][4];
    auto &acc = sum[0];
#pragma unroll
    for (int n = 0; n < D / 8; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    float ls[2], dl[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int qi = q0 + m0 + g + 8 * r;
        ls[r] = qi < T ? lse2[(int64_t)h * T + qi] : INFINITY;      // rows beyond T: P = 0
        dl[r] = qi < T ? delta[(int64_t)h * T + qi] : 0.f;
    }
    const float scale = rsqrtf((float)D);
    if (WK > 1) {      // the tiles that every group reads were fetched by all of them
        cp_wait<0>();
        __syncthreads();
    }
    for (int jt = grp, buf = 0; jt <= it; jt += WK, buf ^= 1) {
        fetch(jt + WK, buf ^ 1);
        cp_wait<1>();
        bwd_group_sync<WK>(grp);
        const uint32_t ks = kv + buf * 2 * kTile, vs = ks + kTile;
        float s[BK / 8][4], dp[BK / 8][4];
#pragma unroll
        for (int n = 0; n < BK / 8; n++) {
            s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
            dp[n][0] = dp[n][1] = dp[n][2] = dp[n][3] = 0.f;
        }
#pragma unroll
        for (int kk = 0; kk < D / 16; kk++) {
            uint32_t aq[4], ad[4];
            ldsm4(a_mk(qs, SD, m0, kk * 16, lane), aq);
            ldsm4(a_mk(dos, SD, m0, kk * 16, lane), ad);
#pragma unroll
            for (int n = 0; n < BK / 8; n += 2) {
                uint32_t bk[4], bv[4];
                ldsm4(b_nk(ks, SD, n * 8, kk * 16, lane), bk);
                ldsm4(b_nk(vs, SD, n * 8, kk * 16, lane), bv);
                mma16<T16>(s[n], aq, bk[0], bk[1]);
                mma16<T16>(s[n + 1], aq, bk[2], bk[3]);
                mma16<T16>(dp[n], ad, bv[0], bv[1]);
                mma16<T16>(dp[n + 1], ad, bv[2], bv[3]);
            }
        }
        uint32_t ds[BK / 16][4];
#pragma unroll
        for (int n = 0; n < BK / 8; n++) {
            float e[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const bool ok = jt < it || n * 8 + 2 * t4 + (c & 1) <= m0 + g + 8 * (c >> 1);      // the diagonal tile is masked
                e[c] = ok ? ex2(s[n][c] - ls[c >> 1]) * (dp[n][c] - dl[c >> 1]) * scale : 0.f;
            }
            ds[n >> 1][(n & 1) * 2] = pk<T16>(e[0], e[1]);
            ds[n >> 1][(n & 1) * 2 + 1] = pk<T16>(e[2], e[3]);
        }
#pragma unroll
        for (int kk = 0; kk < BK / 16; kk++) {
#pragma unroll
            for (int n = 0; n < D / 8; n += 2) {
                uint32_t b[4];
                ldsm4t(b_kn(ks, SD, n * 8, kk * 16, lane), b);
                mma16<T16>(acc[n], ds[kk], b[0], b[1]);
                mma16<T16>(acc[n + 1], ds[kk], b[2], b[3]);
            }
        }
        bwd_group_sync<WK>(grp);      // the tile's buffer is free
    }
    cp_wait<0>();
    float *st[WK];
#pragma unroll
    for (int x = 0; x < WK; x++) st[x] = reinterpret_cast<float *>(smem + (2 + 4 * x) * kTile);
    if (!bwd_join<WK, 1>(sum, st, grp, m0, g, t4)) return;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int qi = q0 + m0 + g + 8 * r;
        if (qi >= T) continue;
        float *dst = dq + (int64_t)qi * ldq + h * D;
#pragma unroll
        for (int n = 0; n < D / 8; n++) *reinterpret_cast<float2 *>(dst + n * 8 + 2 * t4) = make_float2(acc[n][2 * r], acc[n][2 * r + 1]);
    }
}

// dk, dv of one key tile for one query head, summed over the query tiles i >= j, into the per-head workspace
// wk, wv [heads_q, T, head_dim]; a warp owns 16 keys and works on the transposed scores (rows = keys, columns = queries)
template <typename T16, int WK>
__device__ __forceinline__ void attn_bwd_dkv_block(const uint16_t *__restrict__ d_out, const uint16_t *__restrict__ q, const uint16_t *__restrict__ k,
                                                   const uint16_t *__restrict__ v, const float *__restrict__ lse2, const float *__restrict__ delta,
                                                   float *__restrict__ wk, float *__restrict__ wv, int T, int HQ, int HK, int h, int jt) {
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x, grp = tid / kGrp, gt = tid - grp * kGrp, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int kh = h / (HQ / HK), k0 = jt * BK, m0 = (gt >> 5) * 16;
    const int64_t ldq = (int64_t)HQ * D, ldk = (int64_t)HK * D;
    const uint32_t ks = smem_u32(smem), vs = ks + kTile, qo = ks + (2 + 4 * grp) * kTile;      // Q0, dO0, Q1, dO1
    const uint32_t stat = ks + (2 + 4 * WK) * kTile + grp * 4 * BK * 4;            // per buffer: lse [64], delta [64]
    const float *statp = reinterpret_cast<const float *>(smem + (2 + 4 * WK) * kTile + grp * 4 * BK * 4);
    const int n_qt = (T + BK - 1) / BK;
    auto fetch = [&](int it, int buf) {
        if (it < n_qt) {
            fetch_tile<BK, kGrp>(q, ldq, h * D, it * BK, T, qo + buf * 2 * kTile, gt);
            fetch_tile<BK, kGrp>(d_out, ldq, h * D, it * BK, T, qo + (buf * 2 + 1) * kTile, gt);
            const int t = it * BK + (gt & 63);
            const bool live = t < T;
            cp4(stat + (buf * 2 * BK + gt) * 4, (gt < BK ? lse2 : delta) + (int64_t)h * T + (live ? t : 0), live);
        }
        cp_commit();
    };
    fetch_tile<BK, WK * kGrp>(k, ldk, kh * D, k0, T, ks, tid);
    fetch_tile<BK, WK * kGrp>(v, ldk, kh * D, k0, T, vs, tid);
    fetch(jt + grp, 0);
    float sum[2][D / 8][4];
    auto &ak = sum[0];
    auto &av = sum[1];
#pragma unroll
    for (int n = 0; n < D / 8; n++) {
        ak[n][0] = ak[n][1] = ak[n][2] = ak[n][3] = 0.f;
        av[n][0] = av[n][1] = av[n][2] = av[n][3] = 0.f;
    }
    const float scale = rsqrtf((float)D);
    if (WK > 1) {      // the tiles that every group reads were fetched by all of them
        cp_wait<0>();
        __syncthreads();
    }
    for (int it = jt + grp, buf = 0; it < n_qt; it += WK, buf ^= 1) {
        const int q0 = it * BK;
        fetch(it + WK, buf ^ 1);
        cp_wait<1>();
        bwd_group_sync<WK>(grp);
        const uint32_t qs = qo + buf * 2 * kTile, dos = qs + kTile;
        const float *st = statp + buf * 2 * BK;
        const bool masked = it == jt || q0 + BK > T;      // the diagonal tile, and queries beyond T
        uint32_t pf[BK / 16][4], ds[BK / 16][4];
        // 32 queries at a time: the accumulators of dk and dv leave room for half a tile's scores
#pragma unroll
        for (int hf = 0; hf < 2; hf++) {
            float s[4][4], dp[4][4];
#pragma unroll
            for (int n = 0; n < 4; n++) {
                s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
                dp[n][0] = dp[n][1] = dp[n][2] = dp[n][3] = 0.f;
            }
#pragma unroll
            for (int kk = 0; kk < D / 16; kk++) {
                uint32_t a[4], av_[4];
                ldsm4(a_mk(ks, SD, m0, kk * 16, lane), a);
                ldsm4(a_mk(vs, SD, m0, kk * 16, lane), av_);
#pragma unroll
                for (int n = 0; n < 4; n += 2) {
                    uint32_t bq[4], bo[4];
                    ldsm4(b_nk(qs, SD, hf * 32 + n * 8, kk * 16, lane), bq);
                    ldsm4(b_nk(dos, SD, hf * 32 + n * 8, kk * 16, lane), bo);
                    mma16<T16>(s[n], a, bq[0], bq[1]);
                    mma16<T16>(s[n + 1], a, bq[2], bq[3]);
                    mma16<T16>(dp[n], av_, bo[0], bo[1]);
                    mma16<T16>(dp[n + 1], av_, bo[2], bo[3]);
                }
            }
#pragma unroll
            for (int n = 0; n < 4; n++) {
                const int col = hf * 32 + n * 8 + 2 * t4;
                const float2 ls = *reinterpret_cast<const float2 *>(st + col), dl = *reinterpret_cast<const float2 *>(st + BK + col);
                float p[4], e[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const int qi = q0 + col + (c & 1), key = k0 + m0 + g + 8 * (c >> 1);
                    const bool ok = !masked || (key <= qi && qi < T);
                    p[c] = ok ? ex2(s[n][c] - ((c & 1) ? ls.y : ls.x)) : 0.f;
                    e[c] = p[c] * (dp[n][c] - ((c & 1) ? dl.y : dl.x)) * scale;
                }
                const int nn = hf * 4 + n;
                pf[nn >> 1][(nn & 1) * 2] = pk<T16>(p[0], p[1]);
                pf[nn >> 1][(nn & 1) * 2 + 1] = pk<T16>(p[2], p[3]);
                ds[nn >> 1][(nn & 1) * 2] = pk<T16>(e[0], e[1]);
                ds[nn >> 1][(nn & 1) * 2 + 1] = pk<T16>(e[2], e[3]);
            }
        }
#pragma unroll
        for (int kk = 0; kk < BK / 16; kk++) {
#pragma unroll
            for (int n = 0; n < D / 8; n += 2) {
                uint32_t bo[4], bq[4];
                ldsm4t(b_kn(dos, SD, n * 8, kk * 16, lane), bo);
                ldsm4t(b_kn(qs, SD, n * 8, kk * 16, lane), bq);
                mma16<T16>(av[n], pf[kk], bo[0], bo[1]);
                mma16<T16>(av[n + 1], pf[kk], bo[2], bo[3]);
                mma16<T16>(ak[n], ds[kk], bq[0], bq[1]);
                mma16<T16>(ak[n + 1], ds[kk], bq[2], bq[3]);
            }
        }
        bwd_group_sync<WK>(grp);
    }
    cp_wait<0>();
    float *sj[WK];
#pragma unroll
    for (int x = 0; x < WK; x++) sj[x] = reinterpret_cast<float *>(smem + (2 + 4 * x) * kTile);
    if (!bwd_join<WK, 2>(sum, sj, grp, m0, g, t4)) return;
    // the query tiles held q * log2(e) / sqrt(D): dk = dS^T q needs the plain q
    const float unscale = 1.0f / (kLog2e * rsqrtf((float)D));
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int ki = k0 + m0 + g + 8 * r;
        if (ki >= T) continue;
        float *dk_ = wk + ((int64_t)h * T + ki) * D, *dv_ = wv + ((int64_t)h * T + ki) * D;
#pragma unroll
        for (int n = 0; n < D / 8; n++) {
            *reinterpret_cast<float2 *>(dk_ + n * 8 + 2 * t4) = make_float2(ak[n][2 * r] * unscale, ak[n][2 * r + 1] * unscale);
            *reinterpret_cast<float2 *>(dv_ + n * 8 + 2 * t4) = make_float2(av[n][2 * r], av[n][2 * r + 1]);
        }
    }
}

// One launch for both halves of the backward: grid (2 * heads, tiles), even blockIdx.x = the dq block of head x / 2, odd =
// its dk, dv block.  blockIdx.y is the tile's rank by length, longest first (the last query tile sees every key tile,
// key tile 0 is seen by every query tile): blocks are handed out rank by rank, head by head, so blocks of 1..n tile steps pack
// the SMs with one short tail.
template <typename T16, int WK>
__global__ void __launch_bounds__(kGrp * WK, 3 - WK) k_attn_bwd(const uint16_t *__restrict__ d_out, const uint16_t *__restrict__ q, const uint16_t *__restrict__ k,
                                                             const uint16_t *__restrict__ v, const float *__restrict__ lse2, const float *__restrict__ delta,
                                                             float *__restrict__ dq, float *__restrict__ wk, float *__restrict__ wv, int T, int HQ, int HK) {
    pdl_wait();
    pdl_trigger();
    const int h = blockIdx.x >> 1, rank = blockIdx.y;
    if (blockIdx.x & 1) attn_bwd_dkv_block<T16, WK>(d_out, q, k, v, lse2, delta, wk, wv, T, HQ, HK, h, rank);
    else attn_bwd_dq_block<T16, WK>(d_out, q, k, v, lse2, delta, dq, T, HQ, HK, h, (int)gridDim.y - 1 - rank);
}

// dk[t, kh, :] = sum over the query heads of group kh of wk[h, t, :] (same for dv), heads in ascending order
__global__ void k_attn_reduce_kv(const float *__restrict__ wk, const float *__restrict__ wv, float *__restrict__ dk, float *__restrict__ dv, int T,
                                 int HQ, int HK) {
    pdl_wait();
    pdl_trigger();
    const int64_t n4 = (int64_t)T * HK * D / 4;
    const int ratio = HQ / HK;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (int64_t)gridDim.x * blockDim.x) {
        const int c4 = (int)(i % (D / 4));
        const int kh = (int)((i / (D / 4)) % HK);
        const int t = (int)(i / ((int64_t)(D / 4) * HK));
        float4 sk = make_float4(0.f, 0.f, 0.f, 0.f), sv = sk;
        for (int h = kh * ratio; h < (kh + 1) * ratio; h++) {
            const float4 a = __ldg(reinterpret_cast<const float4 *>(wk + ((int64_t)h * T + t) * D) + c4);
            const float4 b = __ldg(reinterpret_cast<const float4 *>(wv + ((int64_t)h * T + t) * D) + c4);
            sk.x += a.x; sk.y += a.y; sk.z += a.z; sk.w += a.w;
            sv.x += b.x; sv.y += b.y; sv.z += b.z; sv.w += b.w;
        }
        reinterpret_cast<float4 *>(dk)[i] = sk;
        reinterpret_cast<float4 *>(dv)[i] = sv;
    }
}

PerDeviceOnce g_attn_attr;
template <typename T16>
cudaError_t attn_allow_smem() {
    cudaError_t e = cudaFuncSetAttribute(k_attn_fwd<T16, 8, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem<8, 1>);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_attn_fwd<T16, 4, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem<4, 2>);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_attn_bwd<T16, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdSmem<1>);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_attn_bwd<T16, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBwdSmem<2>);
    return e;
}
int attn_init() {
    GT_CUDA(per_device_once(g_attn_attr, [] {
        cudaError_t a = attn_allow_smem<__nv_bfloat16>();
        return a == cudaSuccess ? attn_allow_smem<__half>() : a;
    }));
    return GT_OK;
}

int check_shape(int T, int HQ, int HK, int Dh, const char *who) {
    if (T <= 0 || HQ <= 0 || HK <= 0) return failf(GT_ERR_INVALID, "%s: bad shape T=%d heads_q=%d heads_kv=%d", who, T, HQ, HK);
    if (Dh != D) return failf(GT_ERR_UNSUPPORTED, "%s: head_dim %d is not supported (128 only)", who, Dh);
    if (HQ % HK != 0) return failf(GT_ERR_INVALID, "%s: heads_q %d is not a multiple of heads_kv %d", who, HQ, HK);
    return GT_OK;
}
size_t a256(size_t n) { return (n + 255) & ~(size_t)255; }

template <typename T16>
int forward16(gt_engine *e, const uint16_t *q, const uint16_t *k, const uint16_t *v, float *out, uint16_t *out16, float *lse, int T, int HQ, int HK) {
    // 128-query tiles where they give every SM a block; below that the chain of key tiles is what counts (4 x 2 against 8 x 1:
    // 15.6 / 19.7 us at 512 tokens and 28 heads, 18.5 / 27.9 at 777 and 8, but 79 / 69 at 1999 and 16)
    const int big = (T + 127) / 128;
    if (big * HQ >= e->sm_count)
        GT_LAUNCH(e, launch_k(k_attn_fwd<T16, 8, 1>, dim3(HQ, big), dim3(256), kFwdSmem<8, 1>, e->stream, q, k, v, out, out16, lse, T, HQ, HK));
    else
        GT_LAUNCH(e, launch_k(k_attn_fwd<T16, 4, 2>, dim3(HQ, (T + 63) / 64), dim3(256), kFwdSmem<4, 2>, e->stream, q, k, v, out, out16, lse, T, HQ, HK));
    return GT_OK;
}
template <typename T16>
int backward16(gt_engine *e, const float *d_out, const uint16_t *q, const uint16_t *k, const uint16_t *v, const float *out, const float *lse, float *dq,
               float *dk, float *dv, float *delta, uint16_t *do16, float *wk, float *wv, int T, int HQ, int HK) {
    GT_LAUNCH(e, launch_k(k_attn_delta<T16>, dim3((T * HQ * 32 + 255) / 256), dim3(256), 0, e->stream, d_out, out, delta, do16, T, HQ));
    // (two groups per block measured 43 -> 36 us at 777 tokens and 8 heads, 217 -> 239 us at 1999 tokens and 16 heads)
    const dim3 grid(2 * HQ, (T + BK - 1) / BK);
    if ((int)(grid.x * grid.y) > 2 * e->sm_count)
        GT_LAUNCH(e, launch_k(k_attn_bwd<T16, 1>, grid, dim3(kGrp), kBwdSmem<1>, e->stream, (const uint16_t *)do16, q, k, v, lse, (const float *)delta, dq, wk, wv, T, HQ, HK));
    else
        GT_LAUNCH(e, launch_k(k_attn_bwd<T16, 2>, grid, dim3(2 * kGrp), kBwdSmem<2>, e->stream, (const uint16_t *)do16, q, k, v, lse, (const float *)delta, dq, wk, wv, T, HQ, HK));
    const int64_t n4 = (int64_t)T * HK * D / 4;
    GT_LAUNCH(e, launch_k(k_attn_reduce_kv, dim3((unsigned)((n4 + 255) / 256)), dim3(256), 0, e->stream, (const float *)wk, (const float *)wv, dk, dv, T, HQ, HK));
    return GT_OK;
}

}  // namespace

namespace gt {

int attention_operands_on_device(gt_engine *e, const float *q, const float *k, const float *v, void *q16, void *k16, void *v16, int T, int HQ, int HK,
                                 float rope_freq_base) {
    const float qscale = kLog2e * (1.0f / sqrtf((float)D));
    uint16_t *a = (uint16_t *)q16, *b = (uint16_t *)k16, *c = (uint16_t *)v16;
    if (e->math_mode == GT_MATH_BF16) GT_LAUNCH(e, launch_k(k_attn_operands<__nv_bfloat16>, dim3(T), dim3(256), 0, e->stream, q, k, v, a, b, c, HQ, HK, rope_freq_base, qscale));
    else GT_LAUNCH(e, launch_k(k_attn_operands<__half>, dim3(T), dim3(256), 0, e->stream, q, k, v, a, b, c, HQ, HK, rope_freq_base, qscale));
    return GT_OK;
}

int attention_forward16_on_device(gt_engine *e, const void *q16, const void *k16, const void *v16, float *out, float *lse, int T, int HQ, int HK, int Dh,
                                  void *out16) {
    int rc = check_shape(T, HQ, HK, Dh, "attention forward");
    if (rc == GT_OK) rc = attn_init();
    if (rc != GT_OK) return rc;
    const uint16_t *q = (const uint16_t *)q16, *k = (const uint16_t *)k16, *v = (const uint16_t *)v16;
    return e->math_mode == GT_MATH_BF16 ? forward16<__nv_bfloat16>(e, q, k, v, out, (uint16_t *)out16, lse, T, HQ, HK)
                                          : forward16<__half>(e, q, k, v, out, (uint16_t *)out16, lse, T, HQ, HK);
}

// scratch of a backward: delta [HQ, T], dO16 [T, HQ, D], the per-query-head dk / dv workspace [HQ, T, D] x 2; and, for the calls
// on fp32 tensors, q16, k16, v16
int attention_backward16_on_device(gt_engine *e, const float *d_out, const void *q16, const void *k16, const void *v16, const float *out, const float *lse,
                                   float *dq, float *dk, float *dv, int T, int HQ, int HK, int Dh) {
    int rc = check_shape(T, HQ, HK, Dh, "attention backward");
    if (rc == GT_OK) rc = attn_init();
    if (rc != GT_OK) return rc;
    const size_t n_delta = a256((size_t)HQ * T * sizeof(float)), n_do = a256((size_t)HQ * T * D * 2), n_w = (size_t)HQ * T * D * sizeof(float);
    GT_CUDA(e->attn.reserve(n_delta + n_do + 2 * n_w));
    char *p = (char *)e->attn.p;
    float *delta = (float *)p, *wk = (float *)(p + n_delta + n_do), *wv = wk + (size_t)HQ * T * D;
    uint16_t *do16 = (uint16_t *)(p + n_delta);
    const uint16_t *q = (const uint16_t *)q16, *k = (const uint16_t *)k16, *v = (const uint16_t *)v16;
    return e->math_mode == GT_MATH_BF16 ? backward16<__nv_bfloat16>(e, d_out, q, k, v, out, lse, dq, dk, dv, delta, do16, wk, wv, T, HQ, HK)
                                        : backward16<__half>(e, d_out, q, k, v, out, lse, dq, dk, dv, delta, do16, wk, wv, T, HQ, HK);
}

// the calls on fp32 tensors: 16-bit copies in engine scratch, then the same kernels
static int operands_in_scratch(gt_engine *e, const float *q, const float *k, const float *v, int T, int HQ, int HK, void **p16) {
    const size_t nq = a256((size_t)T * HQ * D * 2), nk = a256((size_t)T * HK * D * 2);
    GT_CUDA(e->attn16.reserve(nq + 2 * nk));
    p16[0] = e->attn16.p;
    p16[1] = (char *)e->attn16.p + nq;
    p16[2] = (char *)p16[1] + nk;
    return attention_operands_on_device(e, q, k, v, p16[0], p16[1], p16[2], T, HQ, HK, 0.f);
}

}  // namespace gt

extern "C" {

int gt_attention_forward(gt_engine *e, const float *q, const float *k, const float *v, float *out, float *lse, int32_t T, int32_t heads_q,
                         int32_t heads_kv, int32_t head_dim) {
    if (!e || !q || !k || !v || !out || !lse) return failf(GT_ERR_INVALID, "gt_attention_forward: null argument");
    int rc = check_shape(T, heads_q, heads_kv, head_dim, "attention forward");
    if (rc != GT_OK) return rc;
    std::lock_guard<std::mutex> lk(e->mu);
    GT_CUDA(cudaSetDevice(e->device));
    void *p16[3];
    rc = operands_in_scratch(e, q, k, v, T, heads_q, heads_kv, p16);
    return rc != GT_OK ? rc : attention_forward16_on_device(e, p16[0], p16[1], p16[2], out, lse, T, heads_q, heads_kv, head_dim);
}

int gt_attention_backward(gt_engine *e, const float *d_out, const float *q, const float *k, const float *v, const float *out, const float *lse,
                          float *dq, float *dk, float *dv, int32_t T, int32_t heads_q, int32_t heads_kv, int32_t head_dim) {
    if (!e || !d_out || !q || !k || !v || !out || !lse || !dq || !dk || !dv) return failf(GT_ERR_INVALID, "gt_attention_backward: null argument");
    int rc = check_shape(T, heads_q, heads_kv, head_dim, "attention backward");
    if (rc != GT_OK) return rc;
    std::lock_guard<std::mutex> lk(e->mu);
    GT_CUDA(cudaSetDevice(e->device));
    void *p16[3];
    rc = operands_in_scratch(e, q, k, v, T, heads_q, heads_kv, p16);
    return rc != GT_OK ? rc : attention_backward16_on_device(e, d_out, p16[0], p16[1], p16[2], out, lse, dq, dk, dv, T, heads_q, heads_kv, head_dim);
}

int gt_supports_attention(int32_t T, int32_t head_dim) { return (T > 0 && head_dim == D) ? 1 : 0; }

}  // extern "C"
