// Internal launch interface between the translation units of libglaciertune_b200.so.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <mutex>

namespace gt {

// cudaFuncSetAttribute (dynamic shared memory above 48 KB) applies to the CURRENT device only: an engine on a second
// device of the same process needs its own call.  One PerDeviceOnce per kernel (or group of kernels) remembers on
// which devices `fn` has run; thread-safe.
struct PerDeviceOnce {
    std::mutex mu;
    bool done[64] = {};
};
template <typename F>
cudaError_t per_device_once(PerDeviceOnce &st, F &&fn) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return fn();
    std::lock_guard<std::mutex> lk(st.mu);
    if (st.done[dev]) return cudaSuccess;
    e = fn();
    if (e == cudaSuccess) st.done[dev] = true;
    return e;
}

// Device copy of one frozen base tensor.
struct WeightDev {
    int qtype = 0;
    int N = 0, K = 0;             // [out_features, in_features]
    uint8_t *data = nullptr;      // device blocks (K-quants: the layouts of gt_quant.cuh; F32: floats)
    int64_t nbytes = 0;
    int64_t row_bytes = 0;        // K/256 * block bytes when K % 256 == 0, else 0 (flat super-block stream)
    float *bias = nullptr;        // [N] or null
    bool tma_ok = false;          // tensor maps built: rows of whole super-blocks, or pairs of rows
    int pair_hb = 0;              // maps over pairs of rows (in_features % 256 == 128): half super-blocks per row, else 0
    CUtensorMap tm16_f, tm16_b;         // F16: 64-column boxes of 128 rows (forward) / 64 rows (backward)
    CUtensorMap tm_rows;                // 32-bit words over [N, row_bytes / 4], boxes of 16 rows x two Q4_K blocks / one Q6_K block
    CUtensorMap tm_blk_f, tm_blk;       // K-quants: boxes of one super-block x 256 rows (few-token kernel) / x 64 rows
    CUtensorMap tm_half, tm_half_p;     // boxes of half a super-block x 64 rows (or pairs of rows) / x 32 pairs
};

// ---- CUDA-core kernels (gt_fp32_kernels.cu) -------------------------------------------------------------
// zeroes up to any number of buffers (16-byte aligned, sizes multiples of 16) in launches of kClearBufs
struct ClearBuf {
    void *p;
    size_t bytes;
};
constexpr int kClearBufs = 128;
cudaError_t launch_clear(const ClearBuf *bufs, int n, cudaStream_t s);
cudaError_t launch_q4k_repack(uint8_t *blocks, int64_t nblocks, cudaStream_t s);      // in place
cudaError_t launch_q6k_repack(const uint8_t *gguf_blocks, uint8_t *dev_blocks, int64_t nblocks, cudaStream_t s);
cudaError_t launch_dequant_rows(int qt, const uint8_t *w, int K, int64_t row0, int64_t nrows, float *out, cudaStream_t s);
// ---- fp32-accurate GEMMs on exact weights, any type and shape (gt_exact_gemm.cu)
struct ExactGemm {
    int qtype = 0;
    const uint8_t *w = nullptr;
    int backward = 0;                 // 0: out = act W^T + bias + lora (and residual += it); 1: out (+)= act W + lora
    const float *act = nullptr;       // X [T, K] / dY [T, N]
    float *out = nullptr;             // forward: may be null when residual is given
    float *residual = nullptr;        // forward only
    const float *bias = nullptr;      // forward only
    int assign = 0;                   // backward: out is written, not added to
    int T = 0, N = 0, K = 0;
    // rank-r term (optional): scale * lora_act [T, R] * (forward: lora_w = B [R, N]; backward: lora_w^T, A [K, R])
    const float *lora_act = nullptr, *lora_w = nullptr;
    float scale = 0.f;
    int R = 0;
    const int *flag = nullptr;        // device int: 0 leaves the rank-r term out
};
cudaError_t launch_exact_gemm(const ExactGemm &g, int sm_count, cudaStream_t s);

// LoRA (all fp32 arithmetic).  A is [K, R] row-major, B is [R, N] row-major.  Kernels handle ranks
// [r0, r0+16) of R per launch.
// low[T,R] = X*A ; optionally x16[T, ldx16] = round16(X) (r0 == 0 pass only).
cudaError_t launch_lora_low(const float *X, const float *A, float *low, void *x16, int ldx16, int fp16, int T, int K,
                            int R, cudaStream_t s);
// Y[T,N] += scaling * low * B
cudaError_t launch_lora_delta_fp32(const float *low, const float *B, float *Y, float *residual, int T, int N, int R,
                                   float scaling, const int *nonzero_flag, cudaStream_t s);
// One pass over dY: dB += scaling * low^T * dY ; dLow (pre-zeroed) += dY * B^T ; dy16 = round16(dY) (optional).
cudaError_t launch_lora_bwd_dy(const float *dY, const float *low, const float *B, float *dB, float *dLow, void *dy16,
                               int ld16, int fp16, float scaling, int T, int N, int R, cudaStream_t s);
// dA += scaling * X^T * dLow
cudaError_t launch_lora_bwd_x(const float *X, const float *dLow, float *dA, float scaling, int T, int K, int R,
                              cudaStream_t s);
// dX[T,K] += scaling * dLow * A^T
cudaError_t launch_lora_dx_fp32(const float *dLow, const float *A, float *dX, float scaling, int T, int K, int R,
                                cudaStream_t s);
cudaError_t launch_cast16(const float *src, void *dst, int rows, int cols, int ld_dst, int fp16, cudaStream_t s);
// residual += Y
cudaError_t launch_add_inplace(float *dst, const float *src, int64_t n, cudaStream_t s);
// *flag = any(B != 0)
cudaError_t launch_any_nonzero(const float *B, int64_t n, int *flag, cudaStream_t s);
// scratch: 2 doubles on the device
cudaError_t launch_scale_clip(float *g, int64_t n, float pre_scale, double max_norm, double *scratch, cudaStream_t s);
// g *= scale (no norm, no scratch)
cudaError_t launch_scale(float *g, int64_t n, float scale, cudaStream_t s);

// ---- LoRA products on bf16 warp MMAs for the bf16 math mode (gt_lora_tc.cu); same contracts as the fp32 versions,
// except that `low` / `dLow` must be zero on entry (partial sums arrive by atomics).  Adapters of projections that
// share X go through one pass over it; the dY passes of several members are one launch.  x16 / dy16 (may be null)
// receive the 16-bit copies.
struct LoraXaJob {
    const float *A;
    float *low_zeroed;
    int R;
};
struct LoraDyJob {      // dY == nullptr: dy16 already holds bf16(dY) and is read instead (bf16 mode)
    const float *dY, *low, *B;
    float *dB, *dLow_zeroed;
    void *dy16;
    int ld16;
    float scaling;
    int N, R;
};
struct LoraDaJob {
    const float *dLow;
    float *dA;
    float scaling;
    int R;
};
// dst[T, N] = bias[N] (or zero): up to three such fills ride along with a pass (the output of a split-K GEMM)
struct RowFill {
    float *dst;
    const float *bias;
    int N;
};
cudaError_t launch_lora_xa_group(const float *X, const LoraXaJob *jobs, int n, void *x16, int ldx16, int fp16, int T, int K,
                                 const RowFill *fills, int n_fills, cudaStream_t s);
// the same from an input that already exists as bf16 [T, ld16] (K % 8 == 0, 16-byte aligned): no copy is written
cudaError_t launch_lora_xa16_group(const void *X16, int ld16, const LoraXaJob *jobs, int n, int T, int K, const RowFill *fills, int n_fills,
                                   cudaStream_t s);
// the fills alone
cudaError_t launch_fill_group(const RowFill *fills, int n, int T, cudaStream_t s);
cudaError_t launch_lora_dy_group(const LoraDyJob *jobs, int n, int fp16, int T, const RowFill *fills, int n_fills, cudaStream_t s);
// dA from an X that exists as bf16 [T, ld16] (K % 8 == 0, 16-byte aligned)
cudaError_t launch_lora_da16_group(const void *X16, int ld16, const LoraDaJob *jobs, int n, int T, int K, cudaStream_t s);
cudaError_t launch_lora_da_group(const float *X, const LoraDaJob *jobs, int n, int T, int K, cudaStream_t s);

// ---- tcgen05 kernels (gt_umma_gemm.cu) ------------------------------------------------------------------
struct UmmaLaunch {
    const WeightDev *w = nullptr;
    int backward = 0;              // 0: out[T,N] = act[T,K] * W^T ; 1: out[T,K] += act[T,N] * W
    int fp16 = 0;                  // operand format: 0 bf16, 1 fp16
    const void *act16 = nullptr;   // 16-bit activations [T, ld_act]
    int ld_act = 0;
    int act_early = 0;             // member 0: the kernel launched right before does not write act16, and waited for the one that did
                                   // before it let this one start: the main loop need not wait for it
    int T = 0;
    float *out = nullptr;          // fp32 [T, ld_out]
    int ld_out = 0;
    const float *bias = nullptr;   // forward only
    int out_prefilled = 0;         // forward: out already holds bias/zero, accumulate with atomics (split-K)
    int out_assign = 0;            // backward, member 0: out is overwritten ("dX ="); honoured with plain stores when
                                   // splits == 1, otherwise the caller must have cleared out
    // fused LoRA rank-update (optional)
    const float *lora_act = nullptr;    // fp32 [T, R]: X*A (forward) or dY*B^T (backward)
    float lora_scale = 1.f;             // alpha / r, applied when the tile is rounded to 16 bits
    const float *lora_w = nullptr;      // forward: B [R, N]; backward: A [K, R]
    int rank = 0;
    const int *lora_flag = nullptr;     // device int: 0 -> skip the update
    int splits = 1;
    int tok_chunk = 0;                  // tokens per CTA (umma_group_plan); 0: as many as a CTA can take
    int *status = nullptr;              // device int[4]
    void *trace = nullptr;              // optional device int64[12*128] timeline buffer
    // a window of the weight's rows [row_base, row_base + rows) instead of all of them (rows == 0: the whole tensor):
    // the vocabulary tiles of the LM head.  `out` / `act16` then belong to the window (column 0 = row row_base).
    int row_base = 0, rows = 0;
};
int umma_pick_splits(const WeightDev *w, int backward, int T, int sm_count);
// Returns cudaSuccess or an error; `err` receives a description on failure of a non-CUDA kind.
cudaError_t launch_umma_gemm(const UmmaLaunch &L, cudaStream_t s, const char **err);
// The few-token kernel (gt_umma_few.cu): up to 128 tokens, one member per launch, no fused adapter term.
bool umma_few_ok(const UmmaLaunch &L);
// launch_umma_group will serve these members with the few-token kernel; their adapter terms then follow on kernels that
// update the output with plain read-modify-writes, so such a launch must not run beside another one into the same output
bool umma_group_few(const UmmaLaunch *m, int n);
void umma_few_shape(const UmmaLaunch &L, int *tiles, int *units);
cudaError_t launch_umma_few(const UmmaLaunch &L, cudaStream_t s, const char **err);
bool tmap_encode_2d(CUtensorMap *tm, CUtensorMapDataType dt, const void *base, uint64_t d0, uint64_t d1, uint64_t stride1_bytes,
                    uint32_t b0, uint32_t b1, CUtensorMapSwizzle swz);
// Up to three projections in one launch (see gt_umma_gemm.cu); umma_group_ok tells whether they qualify.
bool umma_group_ok(const UmmaLaunch *m, int n);
void umma_group_plan(UmmaLaunch *m, int n, int sm_count, bool dual = false);      // sets splits and tok_chunk
// dual forward (gate | up, SwiGLU product in the epilogue): see umma_dual_ok
struct UmmaDual {
    void *h16 = nullptr;      // 16-bit [T, ld_h16] in the launch's operand format, or null
    int ld_h16 = 0;
};
bool umma_dual_ok(const UmmaLaunch *m, int sm_count);
cudaError_t launch_umma_group(const UmmaLaunch *m, int n, cudaStream_t s, const char **err, const UmmaDual *dual = nullptr);
cudaError_t umma_init_weight_maps(WeightDev *w, const char **err);
bool umma_available();
cudaError_t launch_bounded_wait_selftest(int *status, long long limit_cycles, cudaStream_t s);


// ---- views of the opaque C-ABI handles for translation units outside gt_engine.cu ---------------------------
struct EngineView {
    int device;
    int math_mode;
    int sm_count;
    cudaStream_t stream;
    int *status;       // device int[4], bounded-wait codes of the tensor-core kernels
    void *mutex;       // std::mutex * serialising calls on the engine
};
// ---- weight-streaming forward projections for few tokens (gt_decode.cu): up to three members that share X in one launch,
// bias, rank-r term and (dual: members 0 and 1) SiLU(out_0) * out_1 included.  T <= stream_max_tokens().
struct DecodeMember {
    const WeightDev *w = nullptr;
    float *out = nullptr;                    // [T, N]; may be null in a dual launch
    const float *low = nullptr, *B = nullptr;      // rank-r term: scale * low [T, R] B [R, N]
    float *low_out = nullptr;                // given: low holds launch_low_few's partial sums, and their sum is kept here
    float scale = 0.f;
    int R = 0;
    const int *flag = nullptr;               // device int: 0 leaves the rank-r term out
};
int stream_max_tokens();
bool decode_group_ok(const WeightDev *const *w, int n, bool dual, int T, int sm_count);
// x_early: the kernel launched right before is launch_low_few on the same X (then X is complete when this one starts)
cudaError_t launch_decode(const DecodeMember *m, int n, const float *X, int T, bool x_early, bool dual, float *hidden, int sm_count, int *status,
                          cudaStream_t s);
// X A for up to three adapters as partial sums of low_few_floats() values each, written (not added), exact fp32
size_t low_few_floats(int T, int R);
bool low_few_ok(int T, int R);
cudaError_t launch_low_few(const float *X, const LoraXaJob *jobs, int n, int T, int K, cudaStream_t s);

// ---- layer glue launchers used inside the library (gt_glue.cu)
cudaError_t launch_swiglu_fwd(const float *gate, const float *up, float *hidden, int64_t n, int sm_count, cudaStream_t s);
// hidden = SiLU(gate) * up written as fp32 (hidden, may be null) and as 16-bit (h16: bf16, or fp16 when fp16 != 0) in one
// pass; n % 4 == 0 and 16-byte-aligned pointers
cudaError_t launch_swiglu_fwd16(const float *gate, const float *up, float *hidden_or_null, void *h16, int64_t n, int fp16, int sm_count,
                                cudaStream_t s);
// dGate, dUp as bf16 only (the operands of the gate,up transpose GEMM); n % 4 == 0, 16-byte-aligned inputs
cudaError_t launch_swiglu_bwd16(const float *d_hidden, const float *gate, const float *up, void *d_gate16, void *d_up16, int64_t n, int sm_count,
                                cudaStream_t s);
// one flat segment of an AdamW launch: parameters, gradients and both moments, n elements; flag (optional) is set to 1
// when a parameter of the segment is non-zero after the step (vec is filled in by the launcher)
struct AdamwSeg {
    float *p;
    const float *g;
    float *m, *v;
    int *flag;
    int64_t n;
    int vec;
};
constexpr int kAdamwSegs = 32;      // segments per launch (16 adapters)
cudaError_t launch_adamw(const AdamwSeg *segs, int n, float lr, float beta1, float beta2, float eps, float weight_decay, int step,
                         int sm_count, cudaStream_t s);
cudaError_t launch_swiglu_bwd(const float *d_hidden, const float *gate, const float *up, float *d_gate, float *d_up, int64_t n, int sm_count,
                              cudaStream_t s);

cudaError_t launch_add(const float *a, const float *b, float *out, int64_t n, int sm_count, cudaStream_t s);
cudaError_t launch_rope(float *q, float *k, int T, int heads_q, int heads_kv, int head_dim, float freq_base, float freq_scale, int rope_dim,
                        int inverse, cudaStream_t s);
// (y16 given: the norm goes out as bf16 there and y is not written)
cudaError_t launch_rmsnorm_fwd(const float *x, const float *w, float *y, int T, int H, float eps, cudaStream_t s, void *y16 = nullptr);
// dx = RMSNorm backward (+ residual, which may be null and may alias dx)
cudaError_t launch_rmsnorm_bwd(const float *dy, const float *x, const float *w, const float *residual, float *dx, int T, int H, float eps,
                               cudaStream_t s, void *dx16 = nullptr);
// sum = a + b (sum may alias a or b), y = RMSNorm(sum) * w
cudaError_t launch_rope_bwd16(float *dq, float *dk, const float *dv, void *dq16, void *dk16, void *dv16, int T, int heads_q, int heads_kv,
                              int head_dim, float freq_base, cudaStream_t s);
cudaError_t launch_add_rmsnorm_fwd(const float *a, const float *b, const float *w, float *sum, float *y, int T, int H, float eps, cudaStream_t s,
                                   void *y16 = nullptr);

// ---- launches with programmatic dependent launch (the kernel must call pdl_wait() before touching global memory).
// On by default; environment GT_PDL=0 launches in plain stream order.
bool pdl_enabled();
template <typename... KArgs, typename... Args>
cudaError_t launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

}  // namespace gt
struct gt_engine;
struct gt_weight;
namespace gt {
EngineView engine_view(gt_engine *e);
const WeightDev *weight_view(const gt_weight *w);
int set_last_error(int code, const char *text);     // records the text for gt_last_error(), returns code
int engine_join_comm(gt_engine *e);                 // engine stream waits for gradient exchanges begun on the side stream (lock held)
}  // namespace gt
