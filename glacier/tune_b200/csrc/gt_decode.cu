// Projections of a few tokens (up to 8), bf16 mode: Y_j[T, N_j] = X W_j^T + bias_j + s_j low_j B_j for up to three K-quant
// members that share X, in one launch; gate | up launches can form SiLU(gate) * up as well.  Replaces gemm_q4_k_batch,
// gemm_q6_k_batch and gemm_q4_k_swiglu_batch of the reference at small batch (launched at
// src/Glacier.Tune/Gpu/GpuLoraEngine.Forward.cs:83-183) and the host's rank-r delta (src/Glacier.Tune/Kernels/LoraKernels.cs:57-86).
//
// With a handful of tokens every weight is used a handful of times: the bound is how fast the packed bytes leave HBM, and
// next to it the instructions spent per weight.  A warp multiplies 16 weight rows on m16n8k16 MMAs (weights = A, tokens =
// B):
//   * the quantized integers enter the MMA as they are, dropped into a bf16 bit pattern: 0x4300 | q = 128 + q, exact for the
//     4-bit and the 6-bit quants; no arithmetic per weight;
//   * scale and offset are applied to the fp32 sums of a sub-block (32 weights in Q4_K, 16 in Q6_K) after its MMAs:
//       Q4_K   sum (a q - b) x = a P - (128 a + b) S,    Q6_K   sum a (q - 32) x = a (P - 160 S),
//       P = sum (128 + q) x,  S = sum x
//     (a = d sc, b = dmin m; src/Glacier.Tune/Gpu/Kernels/tune_bwd.cu:209-211,279-289) - the weights enter exactly, only X is
//     rounded to bf16, and S sums the rounded values.  The Q4_K members of a group that also has a Q6_K one take a and b
//     through bf16 like the tensor-core kernels, which serve such a group above 8 tokens: its q and k keep the values they
//     have always had at every token count;
//   * a thread's bytes of a sub-block are its A fragments in natural order, so X lies in shared memory as plain bf16 rows.
//
// One token goes through the same loops on 8-bit integer MMAs (m16n8k32, m16n8k16): the quants are A's bytes without any
// placing (0.4 integer instructions per Q4_K weight instead of 0.9, and that pipe is the limit), X is a 23-bit fixed-point
// number per half super-block, cut into three signed bytes that fill three of the eight B columns - nearer to X than its
// bf16 rounding - and the sums are exact.  They start from the bit pattern of 1.5 * 2^23, so one subtraction makes them floats.
//
// Work split: a CTA owns a run of 16-row tiles, its warps cut the run's (tile, chunk) items into equal contiguous runs and
// keep two tiled TMA copies in flight each (one per item: 16 rows x two Q4_K or one Q6_K super-block).  A warp's sums of a
// tile go to a shared-memory slot; the slots are added in a fixed order - no atomics, no zero-filled output, the same bits
// every run.  Long rows (or many tokens, whose X must fit beside the rings) are cut over the CTAs of a cluster, joined
// through distributed shared memory.  (Dealing the items out one by one, so that the CTA reads its tiles front to back,
// changed nothing.)
//
// The pass that computes low = X A runs before this kernel; with programmatic dependent launch the copies, the staging of
// X and the whole main loop overlap it, and only the epilogue waits.
//
// Measured, one token through a [3584 | 512, 18944] layer (Q4_K, v and down in Q6_K, rank 16; 155 MB): 163 -> 81 us for its
// eight launches.  Before: one launch per Q4_K member plus fills and rank-r kernels, Q6_K on the 128-row tcgen05 kernel
// (23 us a tensor).  gate | up (76 MB) runs at about 4 TB/s; what is left is latency per item (each warp waits for its own
// copies, IPC 0.45) and about 5 us of start and join per launch.
//
// k_low_few: X A for up to three adapters in kLowParts partial sums each, exact fp32, added up by k_decode in a fixed order.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdlib>
#include <cstring>
#include <mutex>

#include "gt_internal.h"
#include "gt_ptx.cuh"
#include "gt_quant.cuh"

namespace gt {
namespace {

constexpr int kMaxT = 8;
constexpr int kQ4Chunk = 2;                                  // super-blocks per item: 288 bytes per row = 32 mod 128, conflict-free
constexpr int kQ4Row = kQ4Chunk * kQ4KBlockBytes, kQ6Row = kQ6KDevBlockBytes;
constexpr int kStage = 16 * kQ4Row;                          // 4608 bytes (a Q6_K item: 3584)
constexpr int kRing = 2;
constexpr int kScratch = 1024;                               // [16 rows][16] floats: Q4_K (a, c) pairs or a alone, Q6_K scales
constexpr int kWarpBytes = kRing * kStage + kScratch;        // (barriers kept apart)
constexpr int kMaxMembers = 3;
constexpr int kLowParts = 32;      // CTAs per adapter of the X A pass

struct Member {
    CUtensorMap tm;                  // 16-row boxes of packed super-blocks
    float *out;                      // [T, N], may be null in a dual launch
    const float *bias, *B;
    const float *low;                // [parts, T, R]: the rank-r activations, summed over `parts` here ...
    float *low_out;                  // ... and kept for a later backward (may be null)
    const int *flag;
    float scale;
    int R, N, qtype, first, tiles;   // first unit of this member, its 16-row tiles
    int parts;
    int round_c;                     // Q4_K: sub-block constants rounded to bf16
};
struct Params {
    Member m[kMaxMembers];
    const float *X;
    float *hidden;                   // dual: SiLU(member 0) * member 1, [T, N]
    int *status;
    int n_members, dual, n_units, T, K, x_early, mixed;
};

__device__ __forceinline__ void mma_z(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
constexpr uint32_t kMagicBits = 0x4B400000u;      // 1.5 * 2^23: adding an integer below 2^22 to the bits adds it to the value
constexpr float kMagic = 12582912.f;
// D = kMagic + A B on bytes (A unsigned, B signed), as floats
__device__ __forceinline__ void imma32(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    uint32_t r[4];
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(kMagicBits));
#pragma unroll
    for (int i = 0; i < 4; i++) d[i] = __uint_as_float(r[i]) - kMagic;
}
__device__ __forceinline__ void imma16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    uint32_t r[4];
    asm volatile("mma.sync.aligned.m16n8k16.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a0), "r"(a1), "r"(b0), "r"(kMagicBits));
#pragma unroll
    for (int i = 0; i < 4; i++) d[i] = __uint_as_float(r[i]) - kMagic;
}
__device__ __forceinline__ void mma_a(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// shared-memory loads through 32-bit addresses (no 64-bit pointer arithmetic in the inner loops)
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t r;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(r) : "r"(a));
    return r;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 r;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(r.x), "=r"(r.y) : "r"(a));
    return r;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 r;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "r"(a));
    return r;
}
__device__ __forceinline__ float4 lds128f(uint32_t a) {
    const uint4 r = lds128(a);
    return make_float4(__uint_as_float(r.x), __uint_as_float(r.y), __uint_as_float(r.z), __uint_as_float(r.w));
}
__device__ __forceinline__ float2 lds64f(uint32_t a) {
    const uint2 r = lds64(a);
    return make_float2(__uint_as_float(r.x), __uint_as_float(r.y));
}
__device__ __forceinline__ float ld_cluster_f32(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
// bytes 0, 1 (resp. 2, 3) of t as a pair of bf16 values 128 + byte
__device__ __forceinline__ uint32_t pair_lo(uint32_t t) { return __byte_perm(t, 0x43434343u, 0x4140u); }
__device__ __forceinline__ uint32_t pair_hi(uint32_t t) { return __byte_perm(t, 0x43434343u, 0x4342u); }

// Shared memory of a CTA: [X: T rows of bf16 / the three byte planes of one token, xld bytes each]
// [512 bytes of zeros][one token: what a half super-block's fixed-point values are multiplied with][S32: sums over 32 values, TP floats each][S16: 160 * (one token: 32 *)
// sums over 16 values, order (block, step, half, quad)][slots][tile sums][s low of every member][first items, mixed types only][warps: ring, scratch][barriers]
struct Layout {
    int xld, zero, xs, s32, s16, slots, sums, low, first, ring, bars, total;
};
template <int TP, int WARPS>
__host__ __device__ inline Layout layout(int T, int nb, int tiles) {
    Layout l;
    int at = 0;
    auto take = [&](int bytes) {
        const int r = at;
        at += (bytes + 127) & ~127;
        return r;
    };
    const bool t1 = TP == 1;
    l.xld = nb * (t1 ? 256 : 512) + 16;
    take((t1 ? 3 : T) * l.xld);
    l.zero = take(512);
    l.xs = take(t1 ? nb * 2 * 4 : 0);
    l.s32 = take(nb * 8 * TP * 4);
    l.s16 = take(nb * 16 * TP * 4);
    l.slots = take((tiles + WARPS) * 16 * T * 4);
    l.sums = take(tiles * 16 * T * 4);
    l.low = take(kMaxMembers * T * 64 * 4);
    l.first = take((tiles + 1) * 4);
    l.ring = take(WARPS * kWarpBytes);
    l.bars = take(WARPS * kRing * 8);
    l.total = at;
    return l;
}

template <bool T1>
struct Shape {
    static constexpr int TP = T1 ? 1 : kMaxT;        // token columns of the S arrays
    static constexpr int WARPS = T1 ? 16 : 12;       // (several tokens: X takes the room of four rings)
};

// grid (clusters, S), cluster (1, S): CTA rank s takes the s-th run of super-blocks of its cluster's tiles
template <bool T1>
__global__ void __launch_bounds__(32 * Shape<T1>::WARPS, 1) k_decode(const __grid_constant__ Params p) {
    constexpr int TP = Shape<T1>::TP, WARPS = Shape<T1>::WARPS, NTHR = 32 * WARPS;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ int abort_flag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    const int S = gridDim.y, rank = blockIdx.y, T = T1 ? 1 : p.T;
    const int blocks = p.K >> 8;
    // runs of an even number of super-blocks (whole Q4_K items), the last one takes what is left
    const int per = ((blocks + S - 1) / S + 1) & ~1;
    const int kb0 = min(blocks, rank * per), nb = min(blocks, kb0 + per) - kb0;
    const int u0 = (int)((int64_t)p.n_units * blockIdx.x / gridDim.x), u1 = (int)((int64_t)p.n_units * (blockIdx.x + 1) / gridDim.x);
    const int tpu = p.dual ? 2 : 1, n_tiles = (u1 - u0) * tpu;
    const Layout L = layout<TP, WARPS>(T, per, n_tiles);
    const uint32_t sb = smem_u32(smem);
    float *slots = reinterpret_cast<float *>(smem + L.slots), *sums = reinterpret_cast<float *>(smem + L.sums);
    int *first = reinterpret_cast<int *>(smem + L.first);
    // tile -> (member, its 16-row tile)
    auto locate = [&](int tl, int &tile) -> int {
        if (p.dual) {
            tile = u0 + (tl >> 1);
            return tl & 1;
        }
        const int u = u0 + tl;
        int mi = 0;
        for (int j = 1; j < p.n_members; j++)
            if (u >= p.m[j].first) mi = j;
        tile = u - p.m[mi].first;
        return mi;
    };
    const int n4 = (nb + kQ4Chunk - 1) / kQ4Chunk;
    auto chunks = [&](int mi) -> int { return p.m[mi].qtype == kTypeQ4K ? n4 : nb; };
    const uint32_t bar0 = sb + L.bars + warp * kRing * 8, ring = sb + L.ring + warp * kWarpBytes, scr = ring + kRing * kStage;
    if (lane == 0) {
        for (int j = 0; j < p.n_members; j++) tma_prefetch_desc(&p.m[j].tm);
        for (int i = 0; i < kRing; i++) mbar_init(bar0 + 8 * i, 1);
        fence_mbar_init();
    }
    if (tid == 0) abort_flag = 0;
    if (tid < 32) *reinterpret_cast<uint4 *>(smem + L.zero + tid * 16) = make_uint4(0u, 0u, 0u, 0u);
    // items before tile tl: closed form where all members have one type, else a table made by a running warp scan
    const int nc_all = chunks(0);
    if (p.mixed) {
        if (warp == 0) {
            int base = 0;
            for (int t0 = 0; t0 < n_tiles; t0 += 32) {
                int tile, c = 0;
                if (t0 + lane < n_tiles) c = chunks(locate(t0 + lane, tile));
                int incl = c;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += v;
                }
                if (t0 + lane < n_tiles) first[t0 + lane] = base + incl - c;
                base += __shfl_sync(0xffffffffu, incl, 31);
            }
            if (lane == 0) first[n_tiles] = base;
        }
        __syncthreads();
    } else {
        __syncwarp();
    }
    auto before = [&](int tl) -> int { return p.mixed ? first[tl] : tl * nc_all; };
    const int n_items = before(n_tiles);
    const int i0 = (int)((int64_t)n_items * warp / WARPS), i1 = (int)((int64_t)n_items * (warp + 1) / WARPS);

    // the warp's next item to issue and to consume: tile (local index, member, 16-row tile) and chunk
    struct Cursor {
        int tl, mi, tile, c, nc;
    };
    auto seek = [&](Cursor &q, int item) {
        int tl = 0;
        if (p.mixed) while (tl + 1 < n_tiles && first[tl + 1] <= item) tl++;
        else tl = item / nc_all;
        q.tl = tl;
        q.mi = locate(tl, q.tile);
        q.nc = chunks(q.mi);
        q.c = item - before(tl);
    };
    auto step = [&](Cursor &q) {
        if (++q.c == q.nc) {
            q.c = 0;
            if (++q.tl < n_tiles) {
                q.mi = locate(q.tl, q.tile);
                q.nc = chunks(q.mi);
            }
        }
    };
    Cursor is, cs;
    if (i0 < i1) seek(is, i0);
    cs = is;
    int is_st = 0;
    auto issue = [&]() {
        if (lane == 0) {
            const Member &M = p.m[is.mi];
            const bool q4 = M.qtype == kTypeQ4K;
            const int words = (q4 ? kQ4KBlockBytes : kQ6KDevBlockBytes) / 4;
            mbar_arrive_expect_tx(bar0 + 8 * is_st, (uint32_t)(16 * (q4 ? kQ4Row : kQ6Row)));
            // (whole boxes are transferred: rows past N and blocks past the row arrive as zeros, a second block that belongs
            // to the next rank is not used)
            tma_load_2d(ring + is_st * kStage, &M.tm, (kb0 + is.c * (q4 ? kQ4Chunk : 1)) * words, is.tile * 16, bar0 + 8 * is_st);
        }
        step(is);
        is_st ^= 1;
    };
    for (int i = i0; i < i1 && i < i0 + kRing; i++) issue();

    // the epilogue's B columns, on their way into L2 while the weights stream
    for (int i = tid + rank * NTHR; i < (u1 - u0) * 16 * tpu; i += NTHR * S) {
        const int tl = i >> 4;
        int tile;
        const Member &M = p.m[locate(tl, tile)];
        const int n = tile * 16 + (i & 15);
        if (n < M.N)
            for (int r = i & 7; r < M.R; r += 8) asm volatile("prefetch.global.L2 [%0];" ::"l"(M.B + (int64_t)r * M.N + (n & ~7)));
    }
    // X comes from the kernel before the one in front of this launch (x_early: that one has waited for it) or from the
    // kernel right before
    if (!p.x_early) pdl_wait();
    pdl_trigger();
    {
        const int nf4 = nb * 64, total = T * nf4;
        constexpr int NB = 4;      // loads in flight per thread
        for (int ib = tid; ib < ((total + 31) & ~31); ib += NB * NTHR) {
            float4 xv[NB];
#pragma unroll
            for (int q = 0; q < NB; q++) {
                const int i = ib + q * NTHR, t = T1 ? 0 : i / nf4, f = T1 ? i : i - t * nf4;
                xv[q] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (i < total) xv[q] = __ldg(reinterpret_cast<const float4 *>(p.X + (int64_t)t * p.K + (int64_t)kb0 * 256) + f);
            }
#pragma unroll
            for (int q = 0; q < NB; q++) {
                const int i = ib + q * NTHR;
                if ((i & ~31) >= total) break;      // (whole warps)
                const bool live = i < total;
                const int t = T1 ? 0 : i / nf4, f = T1 ? i : i - t * nf4;
                const float4 v = xv[q];
                if (T1) {
                    // a warp holds a half super-block: |x| 2^k < 2^22 for the largest of its 128 values
                    const float mx = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
                    const uint32_t e = max(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)) >> 23, 22u);
                    const float up = __uint_as_float((275u - min(e, 254u)) << 23);
                    const float down = e == 255u ? __uint_as_float(0x7FC00000u) : __uint_as_float((e - 21u) << 23);      // inf, nan: nan
                    const int q0 = __float2int_rn(v.x * up), q1 = __float2int_rn(v.y * up), q2 = __float2int_rn(v.z * up), q3 = __float2int_rn(v.w * up);
                    auto bytes = [](int a, int b, int c, int d, uint32_t sel) -> uint32_t {
                        return __byte_perm(__byte_perm(a, b, sel), __byte_perm(c, d, sel), 0x5410u);
                    };
                    int si = q0 + q1 + q2 + q3;
                    si += __shfl_xor_sync(0xffffffffu, si, 1);
                    si += __shfl_xor_sync(0xffffffffu, si, 2);      // 16 values
                    const int si32 = si + __shfl_xor_sync(0xffffffffu, si, 4);
                    if (live) {
                        uint8_t *dst = smem + f * 4;
                        *reinterpret_cast<uint32_t *>(dst) = bytes(q0, q1, q2, q3, 0x0040u);
                        *reinterpret_cast<uint32_t *>(dst + L.xld) = bytes(q0 + 0x80, q1 + 0x80, q2 + 0x80, q3 + 0x80, 0x0051u);
                        *reinterpret_cast<uint32_t *>(dst + 2 * L.xld) = bytes(q0 + 0x8080, q1 + 0x8080, q2 + 0x8080, q3 + 0x8080, 0x0062u);
                        if ((f & 3) == 0) {
                            const int i16 = (f >> 2) & 15;
                            const int pos = (f >> 6) * 16 + (i16 & 8) + (i16 & 1) * 4 + ((i16 >> 1) & 3);
                            *reinterpret_cast<float *>(smem + L.s16 + pos * 4) = 32.f * down * (float)si;
                        }
                        if ((f & 7) == 0) *reinterpret_cast<float *>(smem + L.s32 + (f >> 3) * 4) = down * (float)si32;
                        if ((f & 31) == 0) *reinterpret_cast<float *>(smem + L.xs + (f >> 5) * 4) = down;
                    }
                    continue;
                }
                const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
                const uint32_t w0 = *reinterpret_cast<const uint32_t *>(&lo), w1 = *reinterpret_cast<const uint32_t *>(&hi);
                float s = __uint_as_float(w0 << 16) + __uint_as_float(w0 & 0xFFFF0000u) + __uint_as_float(w1 << 16) + __uint_as_float(w1 & 0xFFFF0000u);
                s += __shfl_xor_sync(0xffffffffu, s, 1);
                s += __shfl_xor_sync(0xffffffffu, s, 2);      // 16 values
                const float s32 = s + __shfl_xor_sync(0xffffffffu, s, 4);
                if (live) {
                    *reinterpret_cast<uint2 *>(smem + t * L.xld + f * 8) = make_uint2(w0, w1);
                    if ((f & 3) == 0) {
                        const int i16 = (f >> 2) & 15;      // step, quad, half -> step, half, quad
                        const int pos = (f >> 6) * 16 + (i16 & 8) + (i16 & 1) * 4 + ((i16 >> 1) & 3);
                        *reinterpret_cast<float *>(smem + L.s16 + (pos * TP + t) * 4) = 160.f * s;
                    }
                    if ((f & 7) == 0) *reinterpret_cast<float *>(smem + L.s32 + ((f >> 3) * TP + t) * 4) = s32;
                }
            }
        }
    }
    __syncthreads();

    float acc[4] = {0.f, 0.f, 0.f, 0.f};      // rows g (0, 1) and g + 8 (2, 3), tokens 2 t4, 2 t4 + 1
    float acc_c = 0.f;                        // one token: what row lane & 15 has to lose, sum c S (Q6_K: sum a 160 S)
    auto flush = [&](int tl) {
        float *dst = slots + (tl + warp) * 16 * T;
        if (T1) {
            const float c = acc_c + __shfl_xor_sync(0xffffffffu, acc_c, 16);
            const float c0 = __shfl_sync(0xffffffffu, c, g), c1 = __shfl_sync(0xffffffffu, c, g + 8);
            // columns 0, 1 (lanes t4 == 0) and 2 (t4 == 1) are the digits 1, 2^8 and 2^16
            float r0 = t4 == 0 ? fmaf(256.f, acc[1], acc[0]) : 65536.f * acc[0], r1 = t4 == 0 ? fmaf(256.f, acc[3], acc[2]) : 65536.f * acc[2];
            r0 += __shfl_xor_sync(0xffffffffu, r0, 1);
            r1 += __shfl_xor_sync(0xffffffffu, r1, 1);
            if (t4 == 0) {
                dst[g] = r0 - c0;
                dst[g + 8] = r1 - c1;
            }
            acc_c = 0.f;
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int t = 2 * t4 + (i & 1);
                if (t < T) dst[(g + (i >> 1) * 8) * T + t] = acc[i];
            }
        }
        acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
    };
    // B column g: token g's row of X (one token: byte plane g), or (columns beyond) one super-block of zeros, whatever the block
    const bool has_x = g < (T1 ? 3 : T);
    const uint32_t xg = sb + (has_x ? (uint32_t)g * L.xld : (uint32_t)L.zero), x_step = has_x ? (T1 ? 256u : 512u) : 0u;
    const uint32_t s32 = sb + L.s32 + (T1 ? 0 : 2 * t4 * 4), s16 = sb + L.s16 + (T1 ? 0 : 2 * t4 * 4);
    bool ok = true;
    int st = 0;
    uint32_t phase = 0;
    for (int i = i0; i < i1; i++) {
        ok = mbar_wait_bounded(bar0 + 8 * st, phase, &abort_flag, p.status, 501);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint32_t stage = ring + st * kStage;
        if (p.m[cs.mi].qtype == kTypeQ4K) {
            const int nblk = min(kQ4Chunk, nb - cs.c * kQ4Chunk);
            for (int bl = 0; bl < nblk; bl++) {
                const int b = cs.c * kQ4Chunk + bl;
                {   // lane (row = lane & 15, half = lane >> 4) turns four (sc, m) pairs of its row into (a, c = 128 a + b)
                    const uint4 h = lds128(stage + (lane & 15) * kQ4Row + bl * kQ4KBlockBytes + kQ4KHdr);
                    const float d = half_bits_to_f32(h.x & 0xFFFFu), dmin = half_bits_to_f32(h.x >> 16);
                    const bool hi = lane >= 16;
                    const uint32_t sc4 = hi ? ((h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u)) : (h.y & 0x3F3F3F3Fu);
                    const uint32_t m4 = hi ? (((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u)) : (h.z & 0x3F3F3F3Fu);
                    float v[8];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        v[2 * q] = d * (float)((sc4 >> (8 * q)) & 255u);
                        v[2 * q + 1] = fmaf(128.f, v[2 * q], dmin * (float)((m4 >> (8 * q)) & 255u));
                    }
                    if (p.m[cs.mi].round_c) {      // w = a' (16 + q) - r with a' = bf16(16 a) / 16, r = bf16(16 a + b)
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const float a = v[2 * q], b_ = v[2 * q + 1] - 128.f * a;
                            const float ar = __bfloat162float(__float2bfloat16_rn(16.f * a)) * 0.0625f;
                            v[2 * q] = ar;
                            v[2 * q + 1] = fmaf(112.f, ar, __bfloat162float(__float2bfloat16_rn(fmaf(16.f, a, b_))));
                        }
                    }
                    __syncwarp();      // the previous block's scales have been read
                    if (T1) {
                        // the offsets' share is summed here, once per row, not by the four lanes that own a row's products:
                        // c = 128 a + b of a sum over 128 + q is b of the sum over q
                        const float4 s = lds128f(sb + L.s32 + (b * 8 + (hi ? 4 : 0)) * 4);
                        const float xs = __uint_as_float(lds32(sb + L.xs + (b * 2 + (hi ? 1 : 0)) * 4));
                        acc_c = fmaf(fmaf(-128.f, v[0], v[1]), s.x, fmaf(fmaf(-128.f, v[2], v[3]), s.y,
                                fmaf(fmaf(-128.f, v[4], v[5]), s.z, fmaf(fmaf(-128.f, v[6], v[7]), s.w, acc_c))));
                        st_shared_v4(scr + (uint32_t)(((lane & 15) * 8 + (hi ? 4 : 0)) * 4), __float_as_uint(v[0] * xs), __float_as_uint(v[2] * xs),
                                     __float_as_uint(v[4] * xs), __float_as_uint(v[6] * xs));
                    } else {
                        const uint32_t dst = scr + (uint32_t)(((lane & 15) * 8 + (hi ? 4 : 0)) * 8);
                        st_shared_v4(dst, __float_as_uint(v[0]), __float_as_uint(v[1]), __float_as_uint(v[2]), __float_as_uint(v[3]));
                        st_shared_v4(dst + 16, __float_as_uint(v[4]), __float_as_uint(v[5]), __float_as_uint(v[6]), __float_as_uint(v[7]));
                    }
                    __syncwarp();
                }
                const uint32_t qa = stage + g * kQ4Row + bl * kQ4KBlockBytes + t4 * 8, qb = qa + 8 * kQ4Row;
                const uint32_t xb = xg + b * x_step + t4 * (T1 ? 8 : 16);
#pragma unroll
                for (int j = 0; j < 4; j++) {      // sub-blocks 2j (low nibbles) and 2j + 1 (high)
                    const uint32_t qo = j * 32 + (j >> 1) * 16;      // (the header sits between the halves)
                    const uint2 ca = lds64(qa + qo), cb = lds64(qb + qo);
                    // (a, c) of the two sub-blocks for rows g and g + 8; one token: a alone
                    float4 sa, sc;
                    if (T1) {
                        const float2 va = lds64f(scr + (g * 8 + 2 * j) * 4), vc = lds64f(scr + ((g + 8) * 8 + 2 * j) * 4);
                        sa = make_float4(va.x, 0.f, va.y, 0.f);
                        sc = make_float4(vc.x, 0.f, vc.y, 0.f);
                    } else {
                        sa = lds128f(scr + (g * 8 + 2 * j) * 8);
                        sc = lds128f(scr + ((g + 8) * 8 + 2 * j) * 8);
                    }
#pragma unroll
                    for (int hn = 0; hn < 2; hn++) {
                        const uint32_t ta0 = (hn ? ca.x >> 4 : ca.x) & 0x0F0F0F0Fu, ta1 = (hn ? ca.y >> 4 : ca.y) & 0x0F0F0F0Fu;
                        const uint32_t tb0 = (hn ? cb.x >> 4 : cb.x) & 0x0F0F0F0Fu, tb1 = (hn ? cb.y >> 4 : cb.y) & 0x0F0F0F0Fu;
                        float P[4];
                        if (T1) {
                            const uint2 x = lds64(xb + (2 * j + hn) * 32);
                            imma32(P, ta0, tb0, ta1, tb1, x.x, x.y);
                        } else {
                            const uint4 x = lds128(xb + (2 * j + hn) * 64);
                            const uint32_t A0[4] = {pair_lo(ta0), pair_lo(tb0), pair_hi(ta0), pair_hi(tb0)};
                            const uint32_t A1[4] = {pair_lo(ta1), pair_lo(tb1), pair_hi(ta1), pair_hi(tb1)};
                            mma_z(P, A0, x.x, x.y);
                            mma_a(P, A1, x.z, x.w);
                        }
                        const float a = hn ? sa.z : sa.x, ca_ = hn ? sa.w : sa.y, b8 = hn ? sc.z : sc.x, cb_ = hn ? sc.w : sc.y;
                        if (T1) {
                            acc[0] = fmaf(a, P[0], acc[0]);
                            acc[1] = fmaf(a, P[1], acc[1]);
                            acc[2] = fmaf(b8, P[2], acc[2]);
                            acc[3] = fmaf(b8, P[3], acc[3]);
                        } else {
                            const float2 s = lds64f(s32 + (b * 8 + 2 * j + hn) * TP * 4);
                            acc[0] = fmaf(a, P[0], fmaf(-ca_, s.x, acc[0]));
                            acc[1] = fmaf(a, P[1], fmaf(-ca_, s.y, acc[1]));
                            acc[2] = fmaf(b8, P[2], fmaf(-cb_, s.x, acc[2]));
                            acc[3] = fmaf(b8, P[3], fmaf(-cb_, s.y, acc[3]));
                        }
                    }
                }
            }
        } else {
            const int b = cs.c;
            {   // lane (row, step = lane >> 4): eight scales of its row, stored in (step, half, quad) order
                const uint4 h = lds128(stage + (lane & 15) * kQ6Row + (lane >> 4) * kQ6KHalf);
                const uint2 s8 = make_uint2(h.x, h.y);
                const float d = half_bits_to_f32(h.z & 0xFFFFu);
                float v[8];      // byte index = quad * 2 + half
#pragma unroll
                for (int q = 0; q < 8; q++) v[q] = d * (float)(int8_t)(((q < 4 ? s8.x : s8.y) >> (8 * (q & 3))) & 255u);
                const uint32_t dst = scr + (uint32_t)(((lane & 15) * 16 + (lane >> 4) * 8) * 4);
                __syncwarp();
                if (T1) {
                    const uint32_t at = sb + L.s16 + (b * 16 + (lane >> 4) * 8) * 4;
                    const float4 s0 = lds128f(at), s1 = lds128f(at + 16);
                    acc_c = fmaf(v[0], s0.x, fmaf(v[2], s0.y, fmaf(v[4], s0.z, fmaf(v[6], s0.w, acc_c))));
                    acc_c = fmaf(v[1], s1.x, fmaf(v[3], s1.y, fmaf(v[5], s1.z, fmaf(v[7], s1.w, acc_c))));
                    const float xs = __uint_as_float(lds32(sb + L.xs + (b * 2 + (lane >> 4)) * 4));
#pragma unroll
                    for (int q = 0; q < 8; q++) v[q] *= xs;
                }
                st_shared_v4(dst, __float_as_uint(v[0]), __float_as_uint(v[2]), __float_as_uint(v[4]), __float_as_uint(v[6]));
                st_shared_v4(dst + 16, __float_as_uint(v[1]), __float_as_uint(v[3]), __float_as_uint(v[5]), __float_as_uint(v[7]));
                __syncwarp();
            }
            const uint32_t ra = stage + g * kQ6Row, rb = ra + 8 * kQ6Row;
            const uint32_t xb = xg + b * x_step + t4 * (T1 ? 4 : 8);
#pragma unroll
            for (int sh = 0; sh < 4; sh++) {      // (step, half): four sub-blocks of 16, quads 0..3
                const int step = sh >> 1, hf = sh & 1;
                const uint32_t lo = 16 + step * kQ6KHalf + hf * 16 + t4 * 4, ho = 80 + step * kQ6KHalf + hf * 16 + t4 * 4;
                const uint32_t la[2] = {lds32(ra + lo), lds32(ra + lo + 32)}, lb[2] = {lds32(rb + lo), lds32(rb + lo + 32)};
                const uint32_t ha = lds32(ra + ho), hb = lds32(rb + ho);
                const float4 fa = lds128f(scr + (g * 16 + sh * 4) * 4), fb = lds128f(scr + ((g + 8) * 16 + sh * 4) * 4);
                const float aa[4] = {fa.x, fa.y, fa.z, fa.w}, bb[4] = {fb.x, fb.y, fb.z, fb.w};
#pragma unroll
                for (int qd = 0; qd < 4; qd++) {
                    const uint32_t l0 = la[qd & 1], l1 = lb[qd & 1];
                    const uint32_t h0 = qd < 2 ? ha << (4 - 2 * qd) : ha >> (2 * qd - 4), h1 = qd < 2 ? hb << (4 - 2 * qd) : hb >> (2 * qd - 4);
                    const uint32_t ta = ((qd < 2 ? l0 : l0 >> 4) & 0x0F0F0F0Fu) | (h0 & 0x30303030u);
                    const uint32_t tb = ((qd < 2 ? l1 : l1 >> 4) & 0x0F0F0F0Fu) | (h1 & 0x30303030u);
                    float P[4];
                    if (T1) {
                        imma16(P, ta, tb, lds32(xb + step * 128 + qd * 32 + hf * 16));
                        acc[0] = fmaf(aa[qd], P[0], acc[0]);
                        acc[1] = fmaf(aa[qd], P[1], acc[1]);
                        acc[2] = fmaf(bb[qd], P[2], acc[2]);
                        acc[3] = fmaf(bb[qd], P[3], acc[3]);
                    } else {
                        const uint32_t A[4] = {pair_lo(ta), pair_lo(tb), pair_hi(ta), pair_hi(tb)};
                        const uint2 x = lds64(xb + (step * 128 + qd * 32 + hf * 16) * 2);
                        mma_z(P, A, x.x, x.y);
                        const float2 s = lds64f(s16 + (b * 16 + sh * 4 + qd) * TP * 4);
                        acc[0] = fmaf(aa[qd], P[0] - s.x, acc[0]);
                        acc[1] = fmaf(aa[qd], P[1] - s.y, acc[1]);
                        acc[2] = fmaf(bb[qd], P[2] - s.x, acc[2]);
                        acc[3] = fmaf(bb[qd], P[3] - s.y, acc[3]);
                    }
                }
            }
        }
        __syncwarp();      // every lane has read the stage: it can be refilled
        if (i + kRing < i1) issue();
        const int tl = cs.tl;
        step(cs);
        if (cs.c == 0 || i + 1 == i1) flush(tl);
        st ^= 1;
        phase ^= st == 0 ? 1u : 0u;
    }
    if (!ok) {
        // a wait gave up (status word written): let copies that were already issued land before the ring is released
        for (int k = 0; k < 64; k++) __nanosleep(2000);
    }
    __syncthreads();

    // a tile's sum over the warps that worked on it, in warp order
    for (int i = tid; i < n_tiles * 16 * T; i += NTHR) {
        const int tl = i / (16 * T), e = i - tl * 16 * T;
        const int f0 = before(tl), f1 = before(tl + 1) - 1;
        float v = 0.f;
        if (f1 >= f0) {
            // warp of item x: the largest w with n_items * w / WARPS <= x
            const int w0 = (int)(((int64_t)(f0 + 1) * WARPS - 1) / n_items), w1 = (int)(((int64_t)(f1 + 1) * WARPS - 1) / n_items);
            // (with fewer items than warps, some warps in between have none and wrote no slot)
            for (int w = w0; w <= w1; w++)
                if (n_items >= WARPS || n_items * (w + 1) / WARPS > n_items * w / WARPS) v += slots[(tl + w) * 16 * T + e];
        }
        sums[i] = v;
    }
    pdl_wait();      // the low-rank activations, and whoever still read or wrote the outputs
    float *low = reinterpret_cast<float *>(smem + L.low);
    for (int j = 0; j < p.n_members; j++) {
        const Member &M = p.m[j];
        const bool on = M.R > 0 && !(M.flag && *M.flag == 0);
        for (int i = tid; i < T * 64; i += NTHR) {
            const int t = i >> 6, r = i & 63;
            float v = 0.f;
            if (M.R > 0 && r < M.R) {
                const float *q = M.low + t * M.R + r;
                if (M.parts == kLowParts) {
#pragma unroll
                    for (int k = 0; k < kLowParts; k++) v += q[k * T * M.R];
                } else {
                    v = q[0];
                }
                if (M.low_out && blockIdx.x == 0 && rank == 0) M.low_out[t * M.R + r] = v;
            }
            low[j * T * 64 + i] = on ? v * M.scale : 0.f;
        }
    }
    if (S > 1) cluster_sync_all();
    else __syncthreads();
    auto value = [&](int tl, int row, int t, int mi, int n) -> float {
        const Member &M = p.m[mi];
        const int e = (tl * 16 + row) * T + t;
        float v = 0.f;
        if (S > 1) {
            const uint32_t a = smem_u32(sums + e);
            for (int s = 0; s < S; s++) v += ld_cluster_f32(mapa_cluster(a, s));
        } else {
            v = sums[e];
        }
        if (M.bias) v += M.bias[n];
        float dlt = 0.f;
        for (int r0 = 0; r0 < M.R; r0 += 16) {      // (low is zero where the adapter is off)
            float b[16];
#pragma unroll
            for (int r = 0; r < 16; r++) b[r] = r0 + r < M.R ? __ldg(M.B + (int64_t)(r0 + r) * M.N + n) : 0.f;
#pragma unroll
            for (int r = 0; r < 16; r++) dlt = fmaf(low[(mi * T + t) * 64 + r0 + r], b[r], dlt);
        }
        return v + dlt;
    };
    const int n_u = u1 - u0;
    for (int i = tid + rank * NTHR; i < n_u * 16 * T; i += NTHR * S) {
        const int row = i & 15, q = i >> 4, t = T1 ? 0 : q % T, u = T1 ? q : q / T;
        int tile;
        const int mi = locate(u * tpu, tile), n = tile * 16 + row;
        if (n >= p.m[mi].N) continue;
        const float a = value(u * tpu, row, t, mi, n);
        if (p.m[mi].out) p.m[mi].out[(int64_t)t * p.m[mi].N + n] = a;
        if (p.dual) {
            const float c = value(u * 2 + 1, row, t, 1, n);
            if (p.m[1].out) p.m[1].out[(int64_t)t * p.m[1].N + n] = c;
            if (p.hidden) p.hidden[(int64_t)t * p.m[0].N + n] = a * (1.0f / (1.0f + expf(-a))) * c;      // SwiGluKernel.cs:13-35
        }
    }
    if (S > 1) cluster_sync_all();      // nobody leaves while a peer still reads its sums
}

// part[p][T, R] = X A over the p-th run of k: grid (kLowParts, adapters); a thread takes four ranks of every (512 / (R / 4))-th
// k, exact fp32.  The decode kernel adds the parts up: one pass over A with a block's loads all in flight at once
// ([18944, 16]: 11 us with the eight CTAs of a cluster that joined their sums here).
constexpr int kLowThreads = 512;
struct LowParams {
    const float *X;
    const float *A[kMaxMembers];
    float *part[kMaxMembers];
    int R[kMaxMembers];
    int T, K;
};
template <int TT>
__global__ void __launch_bounds__(kLowThreads) k_low_few(const LowParams p) {
    __shared__ float red[kLowThreads / 32][TT * 64];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, a = blockIdx.y, rank = blockIdx.x;
    const int R = p.R[a], q4 = R >> 2;      // R is 4, 8, 16, 32 or 64
    const int c4 = tid & (q4 - 1), k_step = kLowThreads / q4;
    const int k0 = (int)((int64_t)p.K * rank / kLowParts), k1 = (int)((int64_t)p.K * (rank + 1) / kLowParts);
    // A is on its way into L2 while the kernel before this one still runs
    for (int64_t i = (int64_t)k0 * R + tid * 32; i < (int64_t)k1 * R; i += kLowThreads * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.A[a] + i));
    pdl_wait();
    pdl_trigger();
    float acc[TT][4];
#pragma unroll
    for (int t = 0; t < TT; t++) acc[t][0] = acc[t][1] = acc[t][2] = acc[t][3] = 0.f;
    const float *A = p.A[a] + c4 * 4;
#pragma unroll(TT == 1 ? 8 : 4)
    for (int k = k0 + tid / q4; k < k1; k += k_step) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(A + (int64_t)k * R));
#pragma unroll
        for (int t = 0; t < TT; t++) {
            const float x = t < p.T ? __ldg(p.X + (int64_t)t * p.K + k) : 0.f;
            acc[t][0] = fmaf(x, v.x, acc[t][0]);
            acc[t][1] = fmaf(x, v.y, acc[t][1]);
            acc[t][2] = fmaf(x, v.z, acc[t][2]);
            acc[t][3] = fmaf(x, v.w, acc[t][3]);
        }
    }
#pragma unroll
    for (int t = 0; t < TT; t++) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float v = acc[t][i];
            for (int o = 16; o >= q4; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (lane < q4) red[warp][t * R + c4 * 4 + i] = v;
        }
    }
    __syncthreads();
    const int n = p.T * R;
    for (int i = tid; i < n; i += kLowThreads) {
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < kLowThreads / 32; w++) v += red[w][i];
        p.part[a][rank * n + i] = v;
    }
}

template <int TT>
cudaError_t launch_low_tt(const LowParams &p, int n, cudaStream_t s) {
    return launch_k(k_low_few<TT>, dim3(kLowParts, n), dim3(kLowThreads), 0, s, p);
}

constexpr int kMaxSmem = 226 * 1024;      // (227 KB per CTA, static variables included)

// Cluster size: the split of the contraction with the fewest super-blocks on the busiest CTA (rows of many super-blocks give
// few tiles per SM: [3584, 18944] is 224 tiles for 148 SMs), two charged per doubling for the join; X of
// a CTA's part and its tiles' slots must fit beside the rings.
struct Plan {
    int S = 0, clusters = 0, smem = 0;      // S == 0: does not fit
};
// clusters of S such CTAs (one per SM) that run at the same time: a cluster lies inside one GPC, so this is less than
// sm_count / S (18 clusters of 8 would take two rounds where 16 fit); looked up once per device and S
template <bool T1>
int max_clusters(int S, int sm_count) {
    static std::mutex mu;
    static int known[64][4];
    int dev = 0;
    if (S == 1 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return sm_count / S;
    const int at = S == 2 ? 0 : S == 4 ? 1 : 2;
    std::lock_guard<std::mutex> lk(mu);
    if (!known[dev][at]) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(1, S);
        cfg.blockDim = dim3(32 * Shape<T1>::WARPS);
        cfg.dynamicSmemBytes = kMaxSmem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1;
        attr[0].val.clusterDim.y = S;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int n = 0;
        cudaError_t ce = cudaFuncSetAttribute(k_decode<T1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
        if (ce == cudaSuccess) ce = cudaOccupancyMaxActiveClusters(&n, k_decode<T1>, &cfg);
        if (ce != cudaSuccess) cudaGetLastError();
        known[dev][at] = (ce == cudaSuccess && n > 0) ? n : sm_count / (2 * S) + 1;
    }
    return known[dev][at];
}
template <bool T1>
Plan plan_t(int T, int K, int n_units, int tpu, int sm_count) {
    const int blocks = K >> 8;
    Plan best;
    int best_cost = 0;
    for (int S = 1, join = 0; S <= 8; S *= 2, join += 2) {
        const int per = ((blocks + S - 1) / S + 1) & ~1;
        if (S > 1 && (S - 1) * per >= blocks) break;      // a rank would be empty
        int clusters = max_clusters<T1>(S, sm_count);
        if (clusters > n_units) clusters = n_units;
        if (clusters < 1) break;
        const int tiles = (n_units + clusters - 1) / clusters * tpu;
        const Layout l = layout<Shape<T1>::TP, Shape<T1>::WARPS>(T, per, tiles);
        if (l.total > kMaxSmem) continue;
        const int cost = tiles * per + join;
        if (!best.S || cost < best_cost) {
            best.S = S;
            best.clusters = clusters;
            best.smem = l.total;
            best_cost = cost;
        }
    }
    return best;
}
Plan plan(int T, int K, int n_units, int tpu, int sm_count) {
    return T == 1 ? plan_t<true>(T, K, n_units, tpu, sm_count) : plan_t<false>(T, K, n_units, tpu, sm_count);
}

template <bool T1>
cudaError_t launch_t(const Params &p, int sm_count, cudaStream_t s) {
    static PerDeviceOnce configured;
    cudaError_t ce = per_device_once(configured, [] { return cudaFuncSetAttribute(k_decode<T1>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem); });
    if (ce != cudaSuccess) return ce;
    const Plan pl = plan_t<T1>(p.T, p.K, p.n_units, p.dual ? 2 : 1, sm_count);
    if (!pl.S) return cudaErrorInvalidConfiguration;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(pl.clusters, pl.S);
    cfg.blockDim = dim3(32 * Shape<T1>::WARPS);
    cfg.dynamicSmemBytes = pl.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    unsigned na = 0;
    if (pl.S > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = 1;
        attr[na].val.clusterDim.y = pl.S;
        attr[na].val.clusterDim.z = 1;
        na++;
    }
    if (pdl_enabled()) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        na++;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    return cudaLaunchKernelEx(&cfg, k_decode<T1>, p);
}

}  // namespace

int stream_max_tokens() {
    static const int v = [] {
        const char *e = getenv("GT_STREAM_MAX_T");
        const int n = e ? atoi(e) : kMaxT;      // one 8-column MMA; from 9 tokens on the few-token tcgen05 kernel takes over
        return n < 0 ? 0 : (n > kMaxT ? kMaxT : n);
    }();
    return v;
}

// every member whole super-blocks per row with maps, few tokens, and a launch shape that fits
bool decode_group_ok(const WeightDev *const *w, int n, bool dual, int T, int sm_count) {
    if (T < 1 || T > stream_max_tokens() || n < 1 || n > kMaxMembers) return false;
    int units = 0;
    for (int j = 0; j < n; j++) {
        if ((w[j]->qtype != kTypeQ4K && w[j]->qtype != kTypeQ6K) || !w[j]->tma_ok || w[j]->pair_hb || w[j]->K != w[0]->K) return false;
        if (!dual || j == 0) units += (w[j]->N + 15) / 16;
    }
    return plan(T, w[0]->K, units, dual ? 2 : 1, sm_count).S > 0;
}

size_t low_few_floats(int T, int R) { return (size_t)kLowParts * T * R; }
bool low_few_ok(int T, int R) { return T >= 1 && T <= kMaxT && (R == 4 || R == 8 || R == 16 || R == 32 || R == 64); }
cudaError_t launch_low_few(const float *X, const LoraXaJob *jobs, int n, int T, int K, cudaStream_t s) {
    LowParams p{};
    p.X = X;
    p.T = T;
    p.K = K;
    for (int j = 0; j < n; j++) {
        p.A[j] = jobs[j].A;
        p.part[j] = jobs[j].low_zeroed;      // (written, not added to)
        p.R[j] = jobs[j].R;
    }
    if (T == 1) return launch_low_tt<1>(p, n, s);
    if (T <= 4) return launch_low_tt<4>(p, n, s);
    return launch_low_tt<8>(p, n, s);
}

cudaError_t launch_decode(const DecodeMember *m, int n, const float *X, int T, bool x_early, bool dual, float *hidden, int sm_count, int *status,
                          cudaStream_t s) {
    Params p;
    memset(&p, 0, sizeof(p));
    p.X = X;
    p.T = T;
    p.K = m[0].w->K;
    p.x_early = x_early ? 1 : 0;
    p.n_members = n;
    p.dual = dual ? 1 : 0;
    p.hidden = hidden;
    p.status = status;
    for (int j = 0; j < n; j++) {
        const WeightDev *w = m[j].w;
        Member &M = p.m[j];
        M.tm = w->tm_rows;
        M.out = m[j].out;
        M.bias = w->bias;
        M.low = m[j].low;
        M.low_out = m[j].low_out;
        M.parts = m[j].low_out ? kLowParts : 1;
        M.B = m[j].B;
        M.flag = m[j].flag;
        M.scale = m[j].scale;
        M.R = (m[j].low && m[j].B) ? m[j].R : 0;
        M.N = w->N;
        M.qtype = w->qtype;
        M.tiles = (w->N + 15) / 16;
        M.first = p.n_units;
        for (int i = 0; i < n; i++) M.round_c |= m[i].w->qtype != kTypeQ4K;
        p.mixed |= w->qtype != m[0].w->qtype;
        if (!dual || j == 0) p.n_units += M.tiles;
    }
    return T == 1 ? launch_t<true>(p, sm_count, s) : launch_t<false>(p, sm_count, s);
}

}  // namespace gt
