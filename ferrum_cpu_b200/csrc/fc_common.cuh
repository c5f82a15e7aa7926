// Shared declarations of libferrum_cuda: error plumbing, the device layout of a Q8_0
// matrix, and the launch wrappers of every kernel file.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <vector>

#include "../../include/ferrum_cuda.h"

namespace fc {

// ---- errors -------------------------------------------------------------------------
int cuda_fail(cudaError_t e, const char* what, const char* file, int line);
int fail(int code, const char* fmt, ...);
const char* g_err_text();   // the calling thread's last error text
extern thread_local int64_t g_launches;

#define FC_CUDA(expr)                                                               \
    do {                                                                            \
        cudaError_t e__ = (expr);                                                   \
        if (e__ != cudaSuccess) return fc::cuda_fail(e__, #expr, __FILE__, __LINE__); \
    } while (0)
#define FC_TRY(expr)                \
    do {                            \
        int rc__ = (expr);          \
        if (rc__ != FC_OK) return rc__; \
    } while (0)
// After a kernel launch: count it and surface launch-configuration errors.
#define FC_LAUNCHED()                \
    do {                             \
        ++fc::g_launches;            \
        FC_CUDA(cudaGetLastError()); \
    } while (0)

// Device pointers a caller hands to the *_dev entry points are read and written with 16-byte
// vector accesses: anything else is refused on the host before a kernel is launched.
inline bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// Test hooks (fc_debug_set_wait_budget): the cycle budget of every bounded device-side wait, and a
// switch that makes the producers of the pipelined kernels withhold their copies (1), or a kernel's second exchange come to nothing
// (2: the hidden units of a decode step's block; in a tensor-core GEMM one of four warps gives up by itself), so that a test can
// make a wait run out without faulting, trapping or hanging anything.
struct DebugKnobs {
    long long wait_cycles = 4000000000LL;   // ~2 s at 1.9 GHz
    int withhold = 0;
    int withhold_scratch = 0;               // 1: CallScratch finds no memory; 2: a model that holds f16 planes finds none for anything else
};
extern DebugKnobs g_debug;

// ---- host helpers shared by the API files (defined in api.cu) ---------------------------
// Owns device allocations until release().
struct Arena {
    std::vector<void*> ptrs;
    int alloc(void** p, size_t bytes) {
        FC_CUDA(cudaMalloc(p, bytes ? bytes : 16));
        ptrs.push_back(*p);
        return FC_OK;
    }
    template <class T>
    int alloc_n(T** p, size_t n) { return alloc((void**)p, n * sizeof(T)); }
    void release() {
        for (void* p : ptrs) cudaFree(p);
        ptrs.clear();
    }
};
// scratch.cu — device memory of one call, taken and given back in the order of its stream. take leaves p null when there is no
// memory; the other failures are errors. A device's pool lives while weights are retained on it.
constexpr uint64_t kScratchKept = (uint64_t)256 << 20;   // what a device's pool keeps between calls
int scratch_retain(int device);
void scratch_release(int device);
struct CallScratch {
    void* p = nullptr;
    int take(int device, size_t bytes, cudaStream_t st);
    CallScratch() = default;
    CallScratch(const CallScratch&) = delete;
    CallScratch& operator=(const CallScratch&) = delete;
    ~CallScratch();
private:
    cudaStream_t st_ = nullptr;
};
// A word of pinned host memory that kernels raise and the host reads without a copy.
struct StatusWord {
    volatile int* host = nullptr;
    int* dev = nullptr;
    int create();
    void destroy();
    int check(const char* what);   // FC_E_TIMEOUT, once, after a kernel raised it
};
struct QMat;
// Makes `device` current; refuses anything but an sm_100 part (there is no other code path).
int select_device(int device);
int upload_f32(Arena& ar, const float* host, size_t n, float** dev, cudaStream_t st);
// Raw GGML Q8_0 rows [N][K/32 x 34 B] -> the device planes of QMat.
int upload_q8(Arena& ar, const void* host, int N, int K, QMat* out, cudaStream_t st);

// ---- device layout of one Q8_0 matrix [N][K] ----------------------------------------
// The 34-byte GGML blocks are split at upload into two planes so that every row starts
// on a 16-byte boundary:
//   qu [N_pad][K]      uint8  = int8 quant XOR 0x80 (i.e. q + 128), K contiguous
//   d  [N_pad][K/32]   f16    block scales; null: levels alone (scale 1), as a packed QWeight keeps them
// Rows N..N_pad-1 are zero scale / 0x80 quants (value 0) so tiles may read them.
struct QMat {
    const uint8_t* qu = nullptr;
    const __half* d = nullptr;
    int N = 0, K = 0, N_pad = 0;
    bool f16_exact = false;   // two f16 planes hold every weight exactly (largest scale x 128 within f16); else unknown
};
constexpr int kRowPad = 128;
// A Q8_0 matrix as two f16 planes [N][K], hi and kRest times the rest, exactly (gemm_f16.cu).
struct F16Mat {
    void *hi = nullptr, *lo = nullptr;
    int N = 0, K = 0;
};

enum Epilogue : int { EPI_NONE = 0, EPI_GELU = 1, EPI_SWIGLU = 2 };

// activation.rs:9-12 (tanh GELU): 0.5 x (1 + tanh(u)) with u = 0.7978846 (x + 0.044715 x^3). Since (1 + tanh(u)) / 2 is the
// logistic function of 2u, that is x / (1 + exp(-2u)): a handful of instructions where tanhf takes some thirty, and
// without the cancellation of 1 + tanh(u) for large negative u. exp2 and the quotient are the 2-ulp hardware forms.
__device__ __forceinline__ float gelu_f(float x) {
    const float K = 0.7978846f;
    const float u = K * (x + 0.044715f * x * x * x);
    return __fdividef(x, 1.0f + exp2f(u * -2.885390082f));   // -2 log2(e)
}

// ---- decode-step device state (one per stream) ----------------------------------------
// The "window" of token_stream.rs lives on the device: ids fed so far and ids waiting to
// be fed, so that a whole greedy generation runs without a host round trip.
struct StepState {
    int pos;       // cache position of the next fed token (== cached_len)
    int fed;       // index in queue of the next token to feed
    int tail;      // number of ids in queue
    int done;      // set when eos was selected: later steps do nothing
    int eos;       // -1: none
    int error;     // non-zero: bad id / cache full seen on device (FC_E_DIM)
    int pad[2];
};

// ---- kernel launchers (each returns FC_OK or FC_E_CUDA) --------------------------------
// repack.cu
// top: a zeroed word, raised to the bits of the largest |scale|.
int launch_repack_q8(const uint8_t* raw, int N, int K, int N_pad, uint8_t* qu, __half* d, unsigned* top, cudaStream_t st);

// gemv_row.cu — one activation row against up to three matrices (q | k | v, gate | up) of the same K. part.d: f16 scales per
// 32 of k, or null with part.xscale [K]: the scale of input index k (then levels alone); EPI_SWIGLU pairs rows (2i, 2i + 1) of one matrix, or row i of two, as (gate, up) and writes
// part[0].out[i] = silu(gate) * up. Launched as a programmatic dependent.
struct GemvPart {
    const uint8_t* qu = nullptr;
    const __half* d = nullptr;
    const float* xscale = nullptr;
    const float* bias = nullptr;
    float* out = nullptr;
    int N = 0;
};
// What becomes of the row on its way into shared memory: nothing (w null), RMSNorm (b null) or LayerNorm.
struct RowNorm {
    const float *w = nullptr, *b = nullptr;
    float eps = 0.0f;
};
// stats (kRowStats entries): per CTA the largest output and the sum of exp(output - largest); *n_stats: CTAs.
constexpr int kRowStats = 1024;
int launch_gemv_row(const GemvPart* parts, int n_parts, int K, const float* x, const RowNorm& norm, const float* residual, int epi,
                    const StepState* state, cudaStream_t st, float2* stats = nullptr, int* n_stats = nullptr);
inline int launch_gemv_row(const QMat& w, const float* x, const RowNorm& norm, const float* bias, const float* residual, int epi,
                           float* out, const StepState* state, cudaStream_t st, float2* stats = nullptr, int* n_stats = nullptr) {
    const GemvPart p = {w.qu, w.d, nullptr, bias, out, w.N};
    return launch_gemv_row(&p, 1, w.K, x, norm, residual, epi, state, st, stats, n_stats);
}

// rows_alone.cu — a caller's own product of one row or few (y rows N apart), on the kernel for its size; M rows need no scratch
// there. The weight's rows are padded to kRowPad. few_rows: whether they are better off there than on the GEMM.
int launch_gemv_alone(const GemvPart& part, int K, const float* x, cudaStream_t st);
bool few_rows(int N, int K, int M);
int launch_rows_alone(GemvPart part, int K, const float* x, int M, cudaStream_t st);

// attn_step.cu — one attention step over the caches, `split` CTAs per query head; ftab null: no rotation. The state and the
// cached rows are read ahead of its wait: some kernel of the step before it has to wait for all of the step before.
// attn_step_split: the CTAs that share a head at long positions (1: it stays with one), and the position from which on that is
// the faster form; either form takes every position.
bool attn_step_covers(int hd, int ctx);
int attn_step_split(int n_q, int hd, int ctx, int* split, int* from);
int launch_attn_step(const float* qkv, int n_q, int n_kv, int hd, int rope_dim, int neox, const float2* ftab, float inv_linear,
                     float* kc, float* vc, int ctx, int split, const StepState* state, float* out, cudaStream_t st);

// block_step.cu — a block of a decode step in two launches, each on the row x + (part[0] + .. + part[n_part - 1] + bias), left in
// x_out (null: nowhere), behind LayerNorm (g, b) or RMSNorm (b null: a Llama block; bias may be null). The attention half leaves parts
// [n_head][d], the MLP half [block_step_slices][d]. The state and the cached rows are read ahead of the wait, as in launch_attn_step.
// `status` (may be null) and the state's error are raised when a bounded wait runs out.
struct BlockRow {
    const float *x, *part, *bias;
    float* x_out;
    const float *g, *b;
    int n_part, d;
    float eps = 1e-5f;
};
// A matrix of such a block: row r lies at r x stride; d: f16 scales per 32 of k, or null with xscale, the scale of input index k.
struct StepMat {
    const uint8_t* qu = nullptr;
    const __half* d = nullptr;
    const float *xscale = nullptr, *bias = nullptr;
    int stride = 1;
};
struct StepRope {
    int half = 0, neox = 0;
    const float2* ftab = nullptr;
    float inv_linear = 1.0f;
};
bool block_step_covers(int d, int n_head, int F, int ctx, bool gated);
int block_step_slices(int F, bool gated);
int launch_attn_half(const BlockRow& r, int n_head, int n_kv, const StepRope& rope, const StepMat (&qkv)[3], const StepMat& out, float* kc, float* vc, int ctx,
                     float* parts, StepState* state, int* status, cudaStream_t st);
int launch_mlp_half(const BlockRow& r, const StepMat (&up)[2] /* up, or gate and up */, const StepMat& down, int F, float* parts, StepState* state, int* status,
                    cudaStream_t st);

// head_row.cu — the product behind those: N logits and, with stats, per CTA the largest and the mass around it (kRowStats entries at most).
// stats[c], c < *n_stats: over the rows of which (row / kHeadSpan) % *n_stats is c.
constexpr int kHeadSpan = 32;
int launch_head_row(const StepMat& w, int N, const BlockRow& r, float* logits, float2* stats, int* n_stats, const StepState* state, cudaStream_t st);

// Windows of rows that share a forward pass: window b holds rows starts[b] .. starts[b + 1] (device array of B + 1), or, with
// starts == nullptr, T rows each. T: rows of the longest.
struct Windows {
    int B = 0, T = 0;
    const int* starts = nullptr;
    __host__ __device__ int begin(int b) const { return starts ? starts[b] : b * T; }
    __host__ __device__ int length(int b) const { return starts ? starts[b + 1] - starts[b] : T; }
};

// An f32 matrix as n bf16 planes whose sum it is: 2 planes hold it to 2^-17 relative (FC_MATH_BF16X3), 3 exactly
// (FC_MATH_FP32). The form in which activations reach the tensor cores. With a scale (a power of two) they are two f16 planes: hi of
// scale times the matrix, and lo times what that leaves; whoever sets it vouches for scale x values within f16's range. kRest is the lo of
// whatever gemm_f16.cu multiplies, weights included: it brings a remainder of 2^-11 up to where hi is, so that elements down to
// 2^-13 keep 2^-23 of themselves (without it, down to 2^-2).
constexpr float kRest = 2048.0f;
struct Planes {
    void* p[3] = {nullptr, nullptr, nullptr};
    int n = 0;
    float scale = 0.0f, lo = kRest;
};
// Planes of n elements out of a call's scratch; scratch.p stays null when there is no memory.
int take_planes(CallScratch& scratch, Planes& x, int planes, size_t n, int device, cudaStream_t st);
// cols (may be null): column k of rows K wide is multiplied by cols[k] first.
int launch_split_planes(const float* x, const Planes& out, size_t n, cudaStream_t st, const float* cols = nullptr, int K = 4);
// gemm_tc.cu — Y[M][N] = X[M][K]·Wᵀ + bias (+GELU / SwiGLU) (+residual[M][N]) on tcgen05 tensor cores, the weight exact, X
// as planes [M][K]. Output: f32 rows y, or (y == nullptr) planes yp for the next GEMM, as many as X has.
// `status` is a device int raised to FC_E_TIMEOUT when a bounded wait runs out. split_k: few rows may split the K range
// over CTAs; without it a row's result does not depend on how many rows share the launch (the scoring forward).
int launch_gemm_q8_tc(const QMat& w, const Planes& x, const float* bias, const float* residual, int epi, float* y, const Planes* yp,
                      int M, int ldy, int* status, cudaStream_t st, bool split_k = true);

// The LM head fused with the statistics of the softmax tail: instead of logits the
// epilogue leaves, per (row, 128-column tile), the tile's largest logit, the sum of exp(logit - that) and the first
// column that attains it in stats [M][ceil(N / 128)] (16-byte records), and the logit of the row's target
// (targets[M], -1: none) in tlogit [M]. launch_score_combine folds the records of a row in tile order into
// ln(max(softmax(row)[target], 1e-12)) (f32 probability, f64 logarithm) and argmax_first(row) == target.
int launch_gemm_q8_tc_score(const QMat& w, const Planes& x, const int* targets, void* stats, float* tlogit, int M, int* status,
                            cudaStream_t st);
int launch_score_combine(const void* stats, const float* tlogit, const int* targets, int M, int n_tiles, int V, double* logprob,
                         uint8_t* is_greedy, cudaStream_t st);

// gemm_f16.cu — the same two entries on weights and activations as f16 planes. row_inv (may be null): 1 / scale of each row of x in
// place of x.scale. Plane output: bf16, or behind GELU f16 of yp->scale. A row's result does not depend on the rows beside it.
int launch_gemm_f16(const F16Mat& w, const Planes& x, const float* row_inv, const float* bias, const float* residual, int epi, float* y, const Planes* yp,
                    int M, int ldy, int* status, cudaStream_t st);
int launch_gemm_f16_score(const F16Mat& w, const Planes& x, const int* targets, void* stats, float* tlogit, int M, int* status, cudaStream_t st);
// x [M][K] as f16 planes scaled row by row (row_inv [M]: 1 / scale) and w as exact f16 planes, in one launch; either may be empty.
// norms (null, or two zeroed words): the bits of the largest square norm of a weight row, and the complement of those of the smallest but 0.
int launch_f16_planes(const float* x, int M, int K, const Planes& out /* its scale does not count */, float* row_inv, const QMat& w, const F16Mat& planes, unsigned* norms,
                      cudaStream_t st);
// Whether a caller's own two-plane product of M rows is better off there.
bool f16_rows(int K, int M);
int launch_split_f16(const float* x, const Planes& out, size_t n, cudaStream_t st);

// api.cu — the matrix and device behind a resident-weight handle.
const QMat* qweight_matrix(const fc_qweight* w, int* device);

// rowops.cu
int launch_embed_step(const QMat& tok, const float* pos_emb, int ctx, const int* queue, StepState* state,
                      float* x, cudaStream_t st);
// pos: each row's position in its window, or null: r % T.
int launch_embed_rows(const QMat& tok, const float* pos_emb, const int* ids, const int* pos, int R, int T, float* x,
                      int* error_flag, cudaStream_t st);
// LayerNorm written as bf16 planes [rows][d] for the tensor-core GEMM. pick (may be null): row i of the output is row pick[i]
// of x.
int launch_layernorm_planes(const float* x, const float* g, const float* b, const int* pick, int rows, int d, const Planes& out,
                            cudaStream_t st);
// Decode tail over logits[V]: softmax statistics, optional probs[V], optional greedy select
// (append to queue) — and always the end-of-step bookkeeping (pos, fed).
// The tail behind a head product with stats: probabilities (probs set) or the greedy pick, then the step's advance.
int launch_step_finish(const float* logits, int V, const float2* stats, int n_stats, int span, float* probs_or_null, int* queue, int queue_cap,
                       StepState* state, cudaStream_t st);
// End-of-step bookkeeping alone (steps that skip the head).
int launch_step_advance_pdl(StepState* state, cudaStream_t st);
int launch_softmax_row(const float* logits, int V, float* probs, cudaStream_t st);
// sample.cu — one draw of sample_with_params on the device; see the kernel for the arguments.
int launch_sample(const float* in, int V, int from_probs, const fc_sampling& prm, const int* recent, int n_recent,
                  unsigned long long* rng_state, int* queue, int queue_cap, StepState* state, int* token_out, cudaStream_t st);

// Per-layer statistics of a window forward (the device-side counterpart of verbose.rs:85-110): one record per layer.
// Linear on a matrix kept in its GGML block format, decoded in the kernel (ggml_linear.cu): y[M][ldy] = [residual +] bias +
// x · dequant(W)ᵀ; rows of the same kind of table decoded by id (ids, or the queue entry at state->fed when ids is null).
int launch_ggml_linear(const fc_ggml_weight* w, const float* x, const float* bias, const float* residual, float* y, int ldy, int M,
                       cudaStream_t st);
int launch_ggml_rows(const fc_ggml_weight* w, const int* ids, StepState* state, const int* queue, int ctx, int R, float* x,
                     int* error_flag, cudaStream_t st);

// Per-row-scale int8 / int4 linear on a packed matrix (rowq.cu): y[M][ldy] = [residual +] bias + x · W; bias and residual may
// be null, residual may be y itself. scratch: three planes of M x K the caller lends (several rows), with the status word of
// the product, or null: the weight's own.
int launch_rowq_linear(fc_rowq* w, const float* x, const float* bias, const float* residual, float* y, int ldy, int M, cudaStream_t st,
                       const Planes* scratch = nullptr, int* status = nullptr);
// The matrix as rows of levels and its input scales, or false (shapes only the packed form covers).
bool rowq_part(const fc_rowq* w, const float* bias, float* out, GemvPart* part);

struct LayerStatsDev {
    float min, max, mean, pad;
    long long nan_count, inf_count, n;
};
size_t layer_stats_scratch_bytes();
// x (f32), or (x == nullptr) bf16 planes whose sum is the value; n elements; scratch: layer_stats_scratch_bytes().
int launch_layer_stats(const float* x, const Planes& planes, size_t n, void* scratch, LayerStatsDev* out, cudaStream_t st);

// attn.cu
// qkv [R][3d] (q | k | v per row), causal within each window.
int launch_attn_prefill(const float* qkv, const Windows& w, int d, int H, float* out, cudaStream_t st);
// Grouped-query forms (llm.rs:305-341): H query heads share KV key/value heads of width hd.
// Decode: q [H*hd], caches [ctx][KV*hd]. Window: q, k, v rows ld floats apart, out rows ldo apart.
int launch_attn_prefill_gqa(const float* q, const float* k, const float* v, const Windows& w, int ld, int H, int KV, int hd,
                            int ldo, float* out, cudaStream_t st);
// attn_tc.cu — the same on tcgen05 (head_dim 64): planes (two or three of bf16, two of f16) of qkv [R][3d] in, as many planes of the
// attention output [R][d] out; `status` is raised on a timeout.
int launch_attn_prefill_tc(const Planes& qkv, const Windows& w, int R, int d, int H, const Planes& out, int* status, cudaStream_t st);
// Grouped-query form: planes [R][(H + 2 KV) * 64] in (q heads | k heads | v heads), [R][H * 64] out.
int launch_attn_prefill_tc_gqa(const Planes& qkv, const Windows& w, int R, int H, int KV, const Planes& out, int* status, cudaStream_t st);

// decode_batch.cu — one lock-step decode step for S <= kBatchMaxStreams streams.
// Fragment-major copy of a Q8_0 matrix for the warp-level tensor-core product: per (16 rows,
// 32-wide block) 512 bytes of biased quants in lane order (q) and 8 pairs of f16 scales (d).
struct QFrag {
    const void* q = nullptr;
    const void* d = nullptr;
    int N = 0, K = 0, N_pad = 0;
};
constexpr int kBatchMaxStreams = 64;
size_t frag_quant_bytes(const QMat& w);
size_t frag_scale_bytes(const QMat& w);
int launch_repack_frag(const QMat& w, void* fq, void* fd, cudaStream_t st);
// Columns of the activation planes for S streams (two f16 rows per stream, padded to the MMA tiling).
int batch_cols(int S);
// Y = X · Wᵀ for S streams. xp: f16 rows [batch_cols(S)][K], row 2s = hi and row 2s + 1 = lo of stream s (rows past
// 2S zero).
// Where the result goes: f32 rows (optionally residual + result; residual may be y) and / or f16 hi / lo rows (after
// bias and epilogue), or raw partial sums part[splits][S][N] of K ranges (no bias; the consumer adds them in order,
// then the bias and the residual).
struct SkinnyOut {
    float* y = nullptr;
    int ldy = 0;
    const float* residual = nullptr;
    void* planes = nullptr;
    int ldp = 0;
    float* part = nullptr;
    int max_warps = 16;   // warps per CTA; 8 when several chains of step kernels share the GPU (two or three CTAs per SM then)
    bool long_k_block = true;   // 32 warps on the 16-row tile for long K (up to 16 streams); off when more than two chains share the GPU
};
int skinny_max_splits();
int launch_skinny_q8(const QFrag& w, int S, const void* xp, const float* bias, int epi, const SkinnyOut& out, int* splits_used,
                     cudaStream_t st);
int launch_embed_batch(const QMat& tok, const float* pos_emb, const int* cur, const int* pos, int S, float* x, cudaStream_t st);
// LayerNorm rows as f16 hi / lo rows; with partials (part != null) the row is first completed, x_new = x + (sum of the
// n_part partial products part[n_part][S][d] + part_bias), and stored to x_out.
int launch_ln_rows_f16(const float* x, const float* part, int n_part, const float* part_bias, float* x_out, const float* g,
                       const float* b, int S, int d, void* xp, cudaStream_t st);
// qkv [S][3d] of this step; kcs / vcs: per-stream cache base pointers (device array), layer_off floats into each.
int launch_attn_decode_batch(const float* qkv, float* const* kcs, float* const* vcs, size_t layer_off, int d, int H, int ctx,
                             const int* pos, int S, void* ap, cudaStream_t st);
int launch_pick_batch(const float* logits, int ldl, int V, int S, int eos, int* cur, int* done, int* n_out, int* out, int out_cap,
                      int* pos, int advance, cudaStream_t st);
int launch_scatter_kv(const float* qkv, float* const* kcs, float* const* vcs, size_t layer_off, int S, int n, int d, cudaStream_t st);
int launch_gather_last_rows(const float* x, int S, int n, int d, float* out, cudaStream_t st);
int launch_batch_init(int S, int pos0, const int* status, int* done, int* n_out, int* cur, int* pos, cudaStream_t st);
int launch_gather_first(int* const* queues, StepState* const* states, int prompt_len, int S, int* cur, int* done, int* n_out,
                        int* out, int out_cap, int* pos, cudaStream_t st);

}  // namespace fc
