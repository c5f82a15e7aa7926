// C ABI of libferrum_cuda: model upload, the standalone Q8_0 linear, windowed scoring and
// the KV-cached decode driver. Host logic above the kernels mirrors, in C++, the Rust items
// cited in include/ferrum_cuda.h.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#include "fc_common.cuh"
#include "mega.cuh"

namespace fc {

// ------------------------------------------------------------------------------- errors
static thread_local char g_err[512] = "";
thread_local int64_t g_launches = 0;
DebugKnobs g_debug;

const char* g_err_text() { return g_err; }
int fail(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof g_err, fmt, ap);
    va_end(ap);
    return code;
}
int cuda_fail(cudaError_t e, const char* what, const char* file, int line) {
    snprintf(g_err, sizeof g_err, "CUDA error %d (%s) at %s:%d in %s", (int)e, cudaGetErrorString(e), file, line, what);
    return FC_E_CUDA;
}

// Refuses anything but a Blackwell data-centre part: there is no other code path.
int select_device(int device) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
        cudaGetLastError();
        return fail(FC_E_CUDA, "no CUDA device is visible: libferrum_cuda has no CPU fallback");
    }
    if (device < 0 || device >= n) return fail(FC_E_ARG, "device %d out of range (0..%d)", device, n - 1);
    int major = 0;
    FC_CUDA(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device));
    if (major != 10) return fail(FC_E_CUDA, "device %d has compute capability %d.x; this library is built for sm_100a only", device, major);
    FC_CUDA(cudaSetDevice(device));
    return FC_OK;
}

int upload_f32(Arena& ar, const float* host, size_t n, float** dev, cudaStream_t st) {
    if (!host) return fail(FC_E_FORMAT, "a required f32 tensor is null");
    FC_TRY(ar.alloc_n(dev, n));
    FC_CUDA(cudaMemcpyAsync(*dev, host, n * sizeof(float), cudaMemcpyHostToDevice, st));
    return FC_OK;
}

// loader/mod.rs:147-154: a matrix is Q8_0 only when its row length is a multiple of 32.
int upload_q8(Arena& ar, const void* host, int N, int K, QMat* out, cudaStream_t st) {
    if (!host) return fail(FC_E_FORMAT, "a required Q8_0 tensor is null");
    if (N <= 0 || K <= 0 || K % 32) return fail(FC_E_FORMAT, "Q8_0 matrix [%d][%d]: row length must be a positive multiple of 32", N, K);
    if (K > 12288) return fail(FC_E_SHAPE, "row length %d exceeds the 12288 supported by the decode GEMV", K);
    const int N_pad = (N + kRowPad - 1) / kRowPad * kRowPad;
    const size_t raw_bytes = (size_t)N * (K / 32) * 34;
    uint8_t* raw = nullptr;
    uint8_t* qu = nullptr;
    __half* d = nullptr;
    const size_t top_at = (raw_bytes + 15) & ~(size_t)15;   // the largest scale's word behind the blocks
    unsigned top = 0;
    FC_CUDA(cudaMalloc((void**)&raw, top_at + 16));
    int rc = ar.alloc_n(&qu, (size_t)N_pad * K);
    if (rc == FC_OK) rc = ar.alloc_n(&d, (size_t)N_pad * (K / 32));
    if (rc == FC_OK && cudaMemcpyAsync(raw, host, raw_bytes, cudaMemcpyHostToDevice, st) != cudaSuccess)
        rc = fail(FC_E_CUDA, "upload of a Q8_0 tensor failed");
    if (rc == FC_OK && cudaMemsetAsync(raw + top_at, 0, 16, st) != cudaSuccess) rc = fail(FC_E_CUDA, "upload of a Q8_0 tensor failed");
    if (rc == FC_OK) rc = launch_repack_q8(raw, N, K, N_pad, qu, d, (unsigned*)(raw + top_at), st);
    if (rc == FC_OK && cudaMemcpyAsync(&top, raw + top_at, sizeof(top), cudaMemcpyDeviceToHost, st) != cudaSuccess)
        rc = fail(FC_E_CUDA, "repack of a Q8_0 tensor failed");
    if (rc == FC_OK && cudaStreamSynchronize(st) != cudaSuccess) rc = fail(FC_E_CUDA, "repack of a Q8_0 tensor failed");
    cudaFree(raw);
    FC_TRY(rc);
    out->qu = qu; out->d = d; out->N = N; out->K = K; out->N_pad = N_pad;
    out->f16_exact = top < 0x5FFFu;                          // up to 511.5, and 511.5 x 128 < 65504
    return FC_OK;
}

// A block's matrices as f16 planes and the scales of the activation planes that meet them (gemm_f16.cu).
struct LayerF16 {
    F16Mat qkv, out, up, down;
    float n1 = 0.0f, heads = 0.0f, att = 0.0f, n2 = 0.0f, hid = 0.0f;   // 0: bf16 planes
};
struct LayerDev {
    QMat qkv, out, up, down;
    LayerF16 f16;
    float *qkv_b, *out_b, *up_b, *down_b, *ln1g, *ln1b, *ln2g, *ln2b;
};

}  // namespace fc

using namespace fc;

struct fc_qweight {
    int device;
    Arena arena;
    QMat w;
    StatusWord status;   // of the products on callers' streams
};

namespace fc {
const QMat* qweight_matrix(const fc_qweight* w, int* device) {
    *device = w->device;
    return &w->w;
}
}  // namespace fc

// Per-CTA parameter tables of the persistent decode kernel for one grid size.
struct MegaTable {
    int grid = 0;
    int bias_pack = 0;
    fc::MegaLayer* layers = nullptr;
};

// Buffers of the lock-step decode of many streams (fc_decode_batch), for up to `cap` streams.
struct BatchCtx {
    Arena arena;                       // step buffers
    Arena frag_arena;                  // fragment-major weight copies, made on first use
    bool frags = false;
    std::vector<fc::QFrag> qkv, out, up, down;
    fc::QFrag head;
    int cap = 0, out_cap = 0;
    float *x = nullptr, *x2 = nullptr, *qkv_f = nullptr, *logits = nullptr;   // the residual stream alternates between x and x2
    float* part = nullptr;             // K-split partial sums of the out- and down-projections [splits][S][d]
    void *xp = nullptr, *ap = nullptr, *hp = nullptr;      // f16 hi / lo rows of LayerNorm output, attention output, GELU output
    int *cur = nullptr, *done = nullptr, *n_out = nullptr, *out_tok = nullptr, *pos = nullptr;
    float **kcs = nullptr, **vcs = nullptr;
    int** queues = nullptr;
    fc::StepState** states = nullptr;
    // one step, and four steps in a row (no gap between graph launches inside them), captured for
    // (graph_S, graph_eos, out_cap, graph_group)
    cudaGraphExec_t graph = nullptr, graph4 = nullptr;
    int graph_S = 0, graph_eos = 0, graph_cap = 0, graph_nodes = 0, graph4_nodes = 0, graph_group = 0;
    // the step graph runs groups of streams as parallel branches: branch g > 0 is captured on side[g - 1]
    std::vector<cudaStream_t> side;
    std::vector<cudaEvent_t> side_done;
    cudaEvent_t fork = nullptr;
};

// One batch of scoring windows on its way: what the host sends and gets back, in pinned memory and on the device. Two of
// them, so that the host prepares and harvests one batch while the GPU works on the other.
struct ScoreSlot {
    char *in_h = nullptr, *in_d = nullptr, *out_h = nullptr, *out_d = nullptr;
    size_t in_cap = 0, out_cap = 0;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr, done = nullptr;
    int picked = 0;                  // scored rows
    // in: ids [R] | positions [R] | window starts [B + 1] | scored rows [picked] | their targets [picked]
    // out: status word (8 bytes) | f64 log-probs [picked] | greedy flags [picked]
    int* status_d() const { return (int*)out_d; }
    double* lp_d() const { return (double*)(out_d + 8); }
    uint8_t* gr_d() const { return (uint8_t*)(out_d + 8 + 8 * (size_t)picked); }
    const double* lp_h() const { return (const double*)(out_h + 8); }
    const uint8_t* gr_h() const { return (const uint8_t*)(out_h + 8 + 8 * (size_t)picked); }
    size_t out_bytes() const { return 8 + 9 * (size_t)picked; }
    int reserve(size_t in_bytes, size_t out_bytes) {
        if (!done) {
            FC_CUDA(cudaEventCreate(&ev0));
            FC_CUDA(cudaEventCreate(&ev1));
            FC_CUDA(cudaEventCreateWithFlags(&done, cudaEventDisableTiming));
        }
        auto grow = [](char** h, char** d, size_t* cap, size_t want) -> int {
            if (want <= *cap) return FC_OK;
            if (*h) cudaFreeHost(*h);
            if (*d) cudaFree(*d);
            *h = *d = nullptr;
            *cap = 0;
            FC_CUDA(cudaMallocHost((void**)h, want));
            FC_CUDA(cudaMalloc((void**)d, want));
            *cap = want;
            return FC_OK;
        };
        FC_TRY(grow(&in_h, &in_d, &in_cap, in_bytes));
        return grow(&out_h, &out_d, &out_cap, out_bytes);
    }
    void release() {
        if (in_h) cudaFreeHost(in_h);
        if (out_h) cudaFreeHost(out_h);
        if (in_d) cudaFree(in_d);
        if (out_d) cudaFree(out_d);
        if (ev0) cudaEventDestroy(ev0);
        if (ev1) cudaEventDestroy(ev1);
        if (done) cudaEventDestroy(done);
        *this = ScoreSlot();
    }
};

struct fc_model {
    fc_config cfg;
    int device;
    cudaStream_t st = nullptr;
    Arena arena;       // weights
    Arena ws_arena;    // prefill workspace
    Arena f16_arena;   // the weights as f16 planes, given back when anything else of the model finds no memory
    QMat tok, head;
    float* pos = nullptr;
    float *lnfg = nullptr, *lnfb = nullptr;
    std::vector<LayerDev> layers;
    bool f16 = false;                          // window forwards run on f16 planes where they have a scale: LayerDev::f16, and
    F16Mat head_f16;
    float lnf_scale = 0.0f;
    // prefill workspace for ws_rows rows
    int ws_rows = 0, ws_planes = 0;
    float *x = nullptr, *qkv = nullptr, *att = nullptr, *logits = nullptr, *probs_d = nullptr;
    int *ids_d = nullptr, *err_d = nullptr;
    ScoreSlot slot[2];
    Planes pn, pqkv, patt, phid;               // bf16 planes of LayerNorm output, qkv, attention output, GELU output
    void* head_stats = nullptr;                // fused head: per (row, 128-column tile) softmax records, 16 B each
    float* head_tlogit = nullptr;              // ... and the logit of each row's target
    int* tc_status = nullptr;                  // raised by a scoring kernel (tensor-core GEMM, attention, row tail) on a timeout
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    float last_score_ms = 0.0f;
    // persistent decode kernel: per-layer parameter table on the device, grid size (0: the
    // model's shape is outside what that kernel supports)
    std::vector<MegaTable> mega_tables;  // [0]: the whole GPU; then halves, quarters, eighths
    float* mega_lnf = nullptr;
    QTile mega_head;                     // tile-major copy of the LM head for the persistent kernel
    int mega_grid = 0;                   // grid of mega_tables[0]
    // streams created by fc_decode_batch, kept for the next call
    std::vector<fc_stream*> pool;
    float last_batch_ms = 0.0f, last_batch_prime_ms = 0.0f;
    // per-layer statistics of the last window forward (fc_model_set_layer_stats)
    int stats_on = 0, stats_n = 0;
    LayerStatsDev* stats_d = nullptr;   // [n_layer + 2]: embedding, every block, final LayerNorm
    void* stats_scratch = nullptr;
    cudaEvent_t ev_prime = nullptr;
    BatchCtx batch;
};

struct fc_stream {
    fc_model* m;
    Arena arena;
    float *kc = nullptr, *vc = nullptr;  // [L][ctx][d]
    float *x = nullptr, *q = nullptr, *att = nullptr, *hid = nullptr, *logits = nullptr, *probs = nullptr;
    int* queue = nullptr;
    int queue_cap = 0;
    StepState* state = nullptr;
    int host_pos = 0;
    cudaGraphExec_t graph[2][2][3] = {};   // [heads with a CTA each, shared ones][one step, kChainSteps steps][mode]
    int graph_nodes[2][2][3] = {};
    long long graph_wait = 0;              // the wait budget and the test hook the graphs were captured with
    int graph_withhold = 0;
    int attn_split = 1, split_from = 0;    // CTAs that share a head from position split_from on
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    float last_decode_ms = 0.0f;
    int* status = nullptr;                 // raised by a kernel of its prime or its steps whose bounded wait ran out
    // persistent decode kernel: exchange buffers, grid barrier word
    float* qkv = nullptr;                  // the step's q | k | v row
    float2* stats = nullptr;               // softmax statistics of its logits
    float *parts_a = nullptr, *parts_m = nullptr;   // what the halves of a block leave to add (block_step.cu); null: shapes it does not cover
    float *partg = nullptr, *x1g = nullptr, *statg = nullptr;
    unsigned* bar = nullptr;
    int attn_splits = 1;
    int mode = FC_DECODE_AUTO;
    // fc_decode_batch: index of the parameter table (grid size) this stream's launches use, and
    // the CUDA stream they go to (null: the model's)
    int table = 0;
    cudaStream_t cs = nullptr;
    cudaEvent_t cs_done = nullptr;
    unsigned long long* rng_d = nullptr;   // xorshift64* state of a sampled generation
    unsigned long long* trace = nullptr;   // phase timeline of the persistent kernel
    int trace_on = 0;
};
static constexpr int kTraceCap = 256;   // timeline entries per CTA

namespace fc {

// ------------------------------------------------------------------------- decode step
enum StepMode { STEP_NOHEAD = 0, STEP_SELECT = 1, STEP_PROBS = 2 };

// Final LayerNorm, head and the selection of a step, on one row.
static StepMat step_mat(const QMat& q, const float* bias = nullptr, int row = 0) {
    return StepMat{q.qu + (size_t)row * q.K, q.d + (size_t)row * (q.K / 32), nullptr, bias ? bias + row : nullptr, 1};
}
// tail: the row as the halves of the last block left it (null: x is whole).
static int launch_head(fc_stream* s, const float* x, int mode, const BlockRow* tail = nullptr) {
    fc_model* m = s->m;
    int n_stats = 0;
    if (tail) FC_TRY(launch_head_row(step_mat(m->head), m->head.N, *tail, s->logits, s->stats, &n_stats, s->state, m->st));
    else FC_TRY(launch_gemv_row(m->head, x, RowNorm{m->lnfg, m->lnfb, 1e-5f}, nullptr, nullptr, EPI_NONE, s->logits, s->state, m->st, s->stats, &n_stats));
    return launch_step_finish(s->logits, m->cfg.vocab, s->stats, n_stats, tail ? kHeadSpan : 0, mode == STEP_PROBS ? s->probs : nullptr, s->queue, s->queue_cap, s->state,
                              m->st);
}

// One token through every block as a chain of dependent launches, five a layer: CachedTransformer::feed (slm/cached.rs:100-125)
// -> TransformerBlock::forward_with_cache (transformer.rs:221-294). LayerNorm is the prologue of the product that reads it,
// bias, GELU and residual are epilogues, and the weights of a kernel are asked for while the one ahead of it runs. The
// embedding starts when everything ahead of it is complete, so the attention may read state and caches early.
static int launch_step(fc_stream* s, int mode, int split) {
    fc_model* m = s->m;
    const fc_config& c = m->cfg;
    cudaStream_t st = m->st;
    const int d = c.d_model, hd = d / c.n_head;
    const size_t layer_stride = (size_t)c.ctx * d;
    FC_TRY(launch_embed_step(m->tok, m->pos, c.ctx, s->queue, s->state, s->x, st));
    if (s->parts_a) {
        // two launches a layer (block_step.cu); what a half leaves to add is added by the next one
        BlockRow r = {s->x, nullptr, nullptr, nullptr, nullptr, nullptr, 0, d};
        for (int l = 0; l < c.n_layer; ++l) {
            const LayerDev& L = m->layers[l];
            r.g = L.ln1g; r.b = L.ln1b;
            r.x_out = l ? s->att : nullptr;                  // the first row is whole as it is
            const StepMat qkv[3] = {step_mat(L.qkv, L.qkv_b), step_mat(L.qkv, L.qkv_b, d), step_mat(L.qkv, L.qkv_b, 2 * d)}, up[2] = {step_mat(L.up, L.up_b), {}};
            FC_TRY(launch_attn_half(r, c.n_head, c.n_head, StepRope(), qkv, step_mat(L.out), s->kc + l * layer_stride, s->vc + l * layer_stride, c.ctx,
                                    s->parts_a, s->state, s->status, st));
            r = {l ? s->att : s->x, s->parts_a, L.out_b, s->q, L.ln2g, L.ln2b, c.n_head, d};
            FC_TRY(launch_mlp_half(r, up, step_mat(L.down), c.d_ff, s->parts_m, s->state, s->status, st));
            r = {s->q, s->parts_m, L.down_b, nullptr, m->lnfg, m->lnfb, block_step_slices(c.d_ff, false), d};
        }
        if (mode == STEP_NOHEAD) return launch_step_advance_pdl(s->state, st);
        return launch_head(s, nullptr, mode, &r);
    }
    for (int l = 0; l < c.n_layer; ++l) {
        const LayerDev& L = m->layers[l];
        FC_TRY(launch_gemv_row(L.qkv, s->x, RowNorm{L.ln1g, L.ln1b, 1e-5f}, L.qkv_b, nullptr, EPI_NONE, s->qkv, s->state, st));
        FC_TRY(launch_attn_step(s->qkv, c.n_head, c.n_head, hd, 0, 0, nullptr, 1.0f, s->kc + l * layer_stride, s->vc + l * layer_stride, c.ctx,
                                split, s->state, s->att, st));
        FC_TRY(launch_gemv_row(L.out, s->att, RowNorm(), L.out_b, s->x, EPI_NONE, s->x, s->state, st));
        FC_TRY(launch_gemv_row(L.up, s->x, RowNorm{L.ln2g, L.ln2b, 1e-5f}, L.up_b, nullptr, EPI_GELU, s->hid, s->state, st));
        FC_TRY(launch_gemv_row(L.down, s->hid, RowNorm(), L.down_b, s->x, EPI_NONE, s->x, s->state, st));
    }
    if (mode == STEP_NOHEAD) return launch_step_advance_pdl(s->state, st);
    return launch_head(s, s->x, mode);
}

static void drop_graphs(fc_stream* s) {
    for (auto& form : s->graph)
        for (auto& set : form)
            for (cudaGraphExec_t& g : set) {
                if (g) cudaGraphExecDestroy(g);
                g = nullptr;
            }
}

// The launch-bound step is captured once per mode into a CUDA graph and replayed; every
// per-step quantity (token, position) is read from device state, so no node is updated.
// pos: the position of the (first) step, which decides how many CTAs a head has.
constexpr int kChainSteps = 8;
static int run_step(fc_stream* s, int mode, int pos, bool several = false) {
    const bool shared = pos + (several ? kChainSteps : 1) > s->split_from;
    if (s->graph_wait != g_debug.wait_cycles || s->graph_withhold != g_debug.withhold) {
        FC_CUDA(cudaStreamSynchronize(s->m->st));
        drop_graphs(s);
        s->graph_wait = g_debug.wait_cycles;
        s->graph_withhold = g_debug.withhold;
    }
    cudaGraphExec_t& graph = s->graph[shared][several][mode];
    int& nodes = s->graph_nodes[shared][several][mode];
    if (!graph) {
        cudaStream_t st = s->m->st;
        cudaGraph_t g = nullptr;
        const int64_t before = g_launches;
        FC_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        int rc = FC_OK;
        for (int i = 0; i < (several ? kChainSteps : 1) && rc == FC_OK; ++i) rc = launch_step(s, mode, shared ? s->attn_split : 1);
        const cudaError_t e = cudaStreamEndCapture(st, &g);
        nodes = (int)(g_launches - before);
        g_launches = before;
        if (rc != FC_OK) { if (g) cudaGraphDestroy(g); return rc; }
        FC_CUDA(e);
        const cudaError_t ei = cudaGraphInstantiate(&graph, g, 0);
        cudaGraphDestroy(g);
        FC_CUDA(ei);
    }
    FC_CUDA(cudaGraphLaunch(graph, s->m->st));
    g_launches += nodes;
    return FC_OK;
}

// n tokens from the queue through the persistent decode kernel in one launch. Steps before
// head_from skip the LM head; head steps select greedily when `select`, and the last step
// leaves its probabilities in s->probs when `probs`.
static int run_mega(fc_stream* s, int n, int head_from, int select, int probs) {
    fc_model* m = s->m;
    const fc_config& c = m->cfg;
    MegaParams p;
    p.L = c.n_layer; p.d = c.d_model; p.H = c.n_head; p.F = c.d_ff; p.T = c.ctx; p.V = c.vocab;
    p.tok = m->tok; p.head = m->mega_head; p.pos = m->pos; p.lnfpack = m->mega_lnf;
    const MegaTable& tab = m->mega_tables[s->table];
    p.layers = tab.layers;
    p.bias_pack = tab.bias_pack;
    p.kc = s->kc; p.vc = s->vc;
    p.qg = s->q; p.attg = s->att; p.partg = s->partg; p.x1g = s->x1g; p.xg = s->x; p.hidg = s->hid;
    p.logits = s->logits; p.statg = s->statg; p.probs = probs ? s->probs : nullptr;
    p.queue = s->queue; p.queue_cap = s->queue_cap; p.state = s->state;
    p.bar = s->bar; p.status = s->status;
    p.n_steps = n; p.head_from = head_from; p.select = select;
    p.attn_splits = std::max(1, std::min(s->attn_splits, tab.grid / c.n_head));
    p.trace = s->trace_on ? s->trace : nullptr;
    p.trace_cap = kTraceCap;
    p.wait_cycles = g_debug.wait_cycles; p.withhold = g_debug.withhold;
    cudaStream_t st = s->cs ? s->cs : m->st;
    if (p.trace) FC_CUDA(cudaMemsetAsync(s->trace, 0, (size_t)m->mega_grid * kTraceCap * sizeof(unsigned long long), st));
    return launch_decode_mega(p, tab.grid, st);
}

// n steps from position pos on, the last one in `last_mode`, the ones before it in `mode`.
static int run_steps(fc_stream* s, int n, int mode, int last_mode, int pos) {
    if (n <= 0) return FC_OK;
    if (s->m->mega_grid > 0 && s->mode != FC_DECODE_PER_KERNEL) {
        const int head_from = mode != STEP_NOHEAD ? 0 : (last_mode != STEP_NOHEAD ? n - 1 : n);
        return run_mega(s, n, head_from, last_mode == STEP_SELECT, last_mode == STEP_PROBS);
    }
    for (int i = 0; i < n; ++i) FC_TRY(run_step(s, i + 1 == n ? last_mode : mode, pos + i));
    return FC_OK;
}

// n steps of a generation from position pos on. Left to itself (FC_DECODE_AUTO) it takes the chain of dependent launches; the persistent kernel where
// it was asked for, and where its timeline was.
static int decode_steps(fc_stream* s, int n, int mode, int pos) {
    if (s->m->mega_grid > 0 && (s->mode == FC_DECODE_PERSISTENT || (s->mode == FC_DECODE_AUTO && s->trace_on))) return run_steps(s, n, mode, mode, pos);
    for (; n >= kChainSteps; n -= kChainSteps, pos += kChainSteps) FC_TRY(run_step(s, mode, pos, true));
    for (int i = 0; i < n; ++i) FC_TRY(run_step(s, mode, pos + i));
    return FC_OK;
}

__global__ void set_state_kernel(StepState* st, int pos, int fed, int tail, int done, int eos, int keep_pos) {
    if (!keep_pos) st->pos = pos;
    st->fed = fed; st->tail = tail; st->done = done; st->eos = eos; st->error = 0;
}
static int set_state(fc_stream* s, int pos, int fed, int tail, int eos, int keep_pos) {
    set_state_kernel<<<1, 1, 0, s->m->st>>>(s->state, pos, fed, tail, 0, eos, keep_pos);
    FC_LAUNCHED();
    return FC_OK;
}

static int read_state(fc_stream* s, StepState* out) {
    int status = 0;
    FC_CUDA(cudaMemcpyAsync(out, s->state, sizeof(StepState), cudaMemcpyDeviceToHost, s->m->st));
    FC_CUDA(cudaMemcpyAsync(&status, s->status, sizeof(int), cudaMemcpyDeviceToHost, s->m->st));
    FC_CUDA(cudaStreamSynchronize(s->m->st));
    if (status != 0) {
        cudaMemsetAsync(s->status, 0, sizeof(int), s->m->st);
        return fail(FC_E_TIMEOUT, "a bounded wait inside the prime or a decode step ran out (status %d)", status);
    }
    return FC_OK;
}

static int check_ids(const fc_model* m, const int32_t* ids, size_t n) {
    for (size_t i = 0; i < n; ++i)
        if (ids[i] < 0 || ids[i] >= m->cfg.vocab)
            return fail(FC_E_DIM, "Token index %d out of bounds for vocab_size %d", ids[i], m->cfg.vocab);
    return FC_OK;
}

// -------------------------------------------------------------------- prefill workspace
// bf16 planes a window forward splits its activations into: 3 hold an f32 exactly (FC_MATH_FP32), 2 to 2^-17 relative
// (FC_MATH_BF16X3, for matrices whose rows are whole 64-wide k-blocks).
static int model_planes(const fc_model* m) {
    const fc_config& c = m->cfg;
    return c.math_mode == FC_MATH_BF16X3 && c.d_model % 64 == 0 && c.d_ff % 64 == 0 ? 2 : 3;
}
// The matrices of a two-plane model as f16 planes, and the scales of the activation planes that meet them. A scale is the largest power of two
// that keeps scale x bound within f16, where the bound holds for every input: a LayerNorm's row has norm at most sqrt(d) max|g| +
// |b|, an element of a product at most the norm of its weight row times that (+ bias), a mixture of value rows and GELU at
// most what goes into them. The 1 % is for rounding.
// One gain, bias or weight row far above the others makes the bound useless to them: what an f16 pair leaves of an element does not shrink
// with it any more below 2^-13 (planes of products, 2^-36 is lost of a scaled element) or 2^-2 (the attention's, 2^-25). A scale is therefore 0,
// and its planes stay bf16 (2^-17 of each element), where an element of the usual size of the least gain, bias or row would not keep 2^-17 with
// some bits to spare: 8 for elements below that size, 4 in the attention. Normal draws of 12 x 768 are 2^20 and 2^13 above the two lines.
// With a matrix that f16 cannot hold the whole model stays on the level GEMM, and so it does where the planes (4 bytes a weight) would take
// more than a quarter of the free memory: three times as much stays free for caches, workspaces and other models, which did with 1.06 bytes a weight
// before there were planes.
static int build_f16(fc_model* m, const fc_weights* w) {
    const fc_config& c = m->cfg;
    const int d = c.d_model, F = c.d_ff;
    bool held = m->head.f16_exact;
    size_t weights = (size_t)c.vocab * d;
    for (const LayerDev& L : m->layers) {
        held = held && L.qkv.f16_exact && L.out.f16_exact && L.up.f16_exact && L.down.f16_exact;
        weights += (size_t)4 * d * d + (size_t)2 * d * F;
    }
    if (!held) return FC_OK;
    void* mem = nullptr;
    constexpr int NORMS = 6;                                         // a layer's words: two each of the query and key, the value and the up rows
    const size_t norms_at = weights * 4, norms_bytes = (size_t)c.n_layer * NORMS * sizeof(unsigned);
    size_t free_bytes = 0, total_bytes = 0;
    FC_CUDA(cudaMemGetInfo(&free_bytes, &total_bytes));
    if (norms_at + norms_bytes > free_bytes / 4) return FC_OK;
    const cudaError_t e = cudaMalloc(&mem, norms_at + norms_bytes);
    if (e == cudaErrorMemoryAllocation) { cudaGetLastError(); return FC_OK; }
    FC_CUDA(e);
    m->f16_arena.ptrs.push_back(mem);
    unsigned* norms_d = (unsigned*)((char*)mem + norms_at);
    FC_CUDA(cudaMemsetAsync(norms_d, 0, norms_bytes, m->st));
    char* at = (char*)mem;
    auto make_rows = [&](const QMat& q, const F16Mat& f, int from, int n, unsigned* norms) -> int {
        const size_t off = (size_t)from * q.K;
        QMat part = q;
        part.qu = q.qu + off; part.d = q.d + off / 32; part.N = n;
        return launch_f16_planes(nullptr, 0, 4, Planes(), nullptr, part, F16Mat{(__half*)f.hi + off, (__half*)f.lo + off, n, q.K}, norms, m->st);
    };
    auto place = [&](const QMat& q) {
        const size_t bytes = (size_t)q.N * q.K * 2;
        const F16Mat f = {at, at + bytes, q.N, q.K};
        at += 2 * bytes;
        return f;
    };
    auto make = [&](const QMat& q, F16Mat* f, unsigned* norms) { *f = place(q); return make_rows(q, *f, 0, q.N, norms); };
    FC_TRY(make(m->head, &m->head_f16, nullptr));
    for (int l = 0; l < c.n_layer; ++l) {
        LayerDev& L = m->layers[l];
        unsigned* nw = norms_d + NORMS * l;
        L.f16.qkv = place(L.qkv);
        FC_TRY(make_rows(L.qkv, L.f16.qkv, 0, 2 * d, nw));
        FC_TRY(make_rows(L.qkv, L.f16.qkv, 2 * d, d, nw + 2));
        FC_TRY(make(L.out, &L.f16.out, nullptr));
        FC_TRY(make(L.up, &L.f16.up, nw + 4));
        FC_TRY(make(L.down, &L.f16.down, nullptr));
    }
    std::vector<unsigned> norms((size_t)c.n_layer * NORMS);
    FC_CUDA(cudaMemcpyAsync(norms.data(), norms_d, norms_bytes, cudaMemcpyDeviceToHost, m->st));
    FC_CUDA(cudaStreamSynchronize(m->st));
    struct Range { double most, least; };                            // of magnitudes; least: of those that are not 0 (infinity: none)
    auto join = [](Range a, Range b) { return Range{std::max(a.most, b.most), std::min(a.least, b.least)}; };
    auto range = [](const float* v, size_t n) {
        Range r = {0.0, INFINITY};
        for (size_t i = 0; i < n; ++i) {
            const double a = v[i] != v[i] ? INFINITY : std::fabs((double)v[i]);
            r.most = std::max(r.most, a);
            if (a > 0) r.least = std::min(r.least, a);
        }
        return r;
    };
    auto rows = [](const unsigned* words) {
        float sq[2];
        const unsigned bits[2] = {words[0], ~words[1]};
        memcpy(sq, bits, sizeof(sq));
        return words[0] ? Range{std::sqrt((double)sq[0]), std::sqrt((double)sq[1])} : Range{0.0, INFINITY};
    };
    auto norm = [](const float* v, size_t n) { double t = 0; for (size_t i = 0; i < n; ++i) t += (double)v[i] * v[i]; return std::sqrt(t); };
    // What a LayerNorm leaves: elements of at most `most`, usually of `least` or more, in a row of norm `all`.
    struct Normed { double most, least, all; };
    const double root = std::sqrt((double)d);
    auto normed = [&](const float* g, const float* b) {
        const Range rg = range(g, d), rb = range(b, d);
        Normed r = {root * rg.most + rb.most, INFINITY, root * rg.most + norm(b, d)};
        for (int i = 0; i < d; ++i) {
            const double usual = std::max(std::fabs((double)g[i]), std::fabs((double)b[i]));
            if (usual > 0) r.least = std::min(r.least, usual);
        }
        return r;
    };
    auto scale = [](double bound, double least, int floor_log2) -> float {
        bound *= 1.01;
        if (!(bound < 1e30)) return 0.0f;                            // NaN too
        const double s = bound > 0 ? std::exp2(std::min(15.0, std::floor(std::log2(65504.0 / bound)))) : 1.0;
        return s * least >= std::exp2((double)floor_log2) ? (float)s : 0.0f;
    };
    constexpr int PRODUCT = -36 + 17 + 8, HEADS = -25 + 17 + 4;
    bool any = false;
    for (int l = 0; l < c.n_layer; ++l) {
        const fc_layer_weights& s = w->layers[l];
        LayerF16& f = m->layers[l].f16;
        const Normed n1 = normed(s.ln1_g, s.ln1_b), n2 = normed(s.ln2_g, s.ln2_b);
        const unsigned* nw = &norms[(size_t)NORMS * l];
        const Range v = rows(nw + 2), heads = join(rows(nw), v), up = rows(nw + 4);
        f.n1 = scale(n1.most, n1.least, PRODUCT);
        f.n2 = scale(n2.most, n2.least, PRODUCT);
        f.heads = scale(heads.most * n1.all + range(s.attn_qkv_b, 3 * (size_t)d).most, heads.least * n1.least, HEADS);
        f.att = scale(v.most * n1.all + range(s.attn_qkv_b + 2 * d, d).most, v.least * n1.least, PRODUCT);
        f.hid = scale(up.most * n2.all + range(s.ffn_up_b, F).most, up.least * n2.least, PRODUCT);
        if (f.n1 == 0.0f) f.heads = 0.0f;                            // the level GEMM writes bf16 planes
        if (f.n2 == 0.0f || f.hid == 0.0f) f.n2 = f.hid = 0.0f;      // each GEMM's GELU leaves planes of its own kind
        any = any || f.n1 != 0.0f || f.att != 0.0f || f.n2 != 0.0f;
    }
    const Normed nf = normed(w->out_norm_g, w->out_norm_b);
    m->lnf_scale = scale(nf.most, nf.least, PRODUCT);
    m->f16 = any || m->lnf_scale != 0.0f;
    if (!m->f16) m->f16_arena.release();
    return FC_OK;
}
// What a model allocates besides. Where there is no memory the planes are given back, and it is tried again: whoever had room for a stream,
// a workspace or a batch without them has it with them. `make` leaves nothing behind when it fails.
template <class Make>
static int with_room(fc_model* m, Make make) {
    const bool starved = m->f16 && g_debug.withhold_scratch == 2;
    const int rc = starved ? fail(FC_E_CUDA, "no memory (test hook)") : make();
    if (rc == FC_OK || !m->f16 || !(starved || cudaGetLastError() == cudaErrorMemoryAllocation)) return rc;
    FC_CUDA(cudaStreamSynchronize(m->st));
    m->f16 = false;
    m->f16_arena.release();
    return make();
}
// Whether the window attention runs on the tensor cores (heads of 64).
static bool tensor_attention(const fc_model* m) { return m->cfg.d_model == m->cfg.n_head * 64; }

static int make_workspace(fc_model* m, int rows, int planes) {
    m->ws_arena.release();
    m->ws_rows = m->ws_planes = 0;
    const fc_config& c = m->cfg;
    const size_t R = rows, d = c.d_model, F = c.d_ff;
    Arena& a = m->ws_arena;
    FC_TRY(a.alloc_n(&m->x, R * d));
    FC_TRY(a.alloc_n(&m->logits, (size_t)m->head.N_pad));   // predict_next
    FC_TRY(a.alloc_n(&m->qkv, R * 3 * d));
    FC_TRY(a.alloc_n(&m->att, R * d));
    FC_TRY(a.alloc_n(&m->ids_d, R));
    FC_TRY(a.alloc_n(&m->err_d, 1));
    FC_TRY(a.alloc_n(&m->probs_d, (size_t)c.vocab));
    auto make = [&](Planes* p, size_t n) -> int {
        for (int i = 0; i < planes; ++i) FC_TRY(a.alloc(&p->p[i], n * 2));
        return FC_OK;
    };
    FC_TRY(make(&m->pn, R * d));
    FC_TRY(make(&m->pqkv, R * 3 * d));
    FC_TRY(make(&m->patt, R * d));
    FC_TRY(make(&m->phid, R * F));
    FC_TRY(a.alloc(&m->head_stats, R * (size_t)((c.vocab + 127) / 128) * 16));
    FC_TRY(a.alloc_n(&m->head_tlogit, R));
    FC_TRY(a.alloc_n(&m->tc_status, 1));
    FC_CUDA(cudaMemsetAsync(m->tc_status, 0, sizeof(int), m->st));
    m->ws_rows = rows;
    m->ws_planes = planes;
    return FC_OK;
}
static int ensure_workspace(fc_model* m, int rows, int planes) {
    if (rows <= m->ws_rows && planes <= m->ws_planes) return FC_OK;
    rows = std::max(rows, m->ws_rows);
    planes = std::max(planes, m->ws_planes);
    FC_CUDA(cudaStreamSynchronize(m->st));
    return with_room(m, [&] { return make_workspace(m, rows, planes); });
}

// Sequential::forward (model.rs:51-71) through every block, on the R rows of `win` (device arrays: their ids, and their
// positions in the window, null: r % T).
// Leaves the residual stream in m->x. Between kernels activations are bf16 planes; only the residual stream is f32.
// split_k: see launch_gemm_q8_tc. f32_qkv: the QKV product is written as f32 rows to m->qkv and on_qkv(layer) is called before the attention.
template <class OnQkv>
static int forward_blocks_with(fc_model* m, const Windows& win, int R, const int* ids, const int* pos, int planes, int* status,
                               bool split_k, bool f32_qkv, OnQkv on_qkv) {
    const fc_config& c = m->cfg;
    const int d = c.d_model, F = c.d_ff;
    cudaStream_t st = m->st;
    const bool tc_attn = tensor_attention(m);
    // f16 planes in the two-plane mode, where they have a scale (never in the f32 mode: two of them are a bit short of an f32)
    const bool f16 = m->f16 && planes == 2;
    m->pqkv.n = m->pn.n = m->patt.n = m->phid.n = planes;
    m->pqkv.lo = 1.0f;                                               // the attention adds both planes' products in one place
    auto product = [&](const QMat& q, const F16Mat& h, const Planes& x, const float* bias, const float* residual, int epi, float* y, const Planes* yp) {
        return x.scale != 0.0f ? launch_gemm_f16(h, x, nullptr, bias, residual, epi, y, yp, R, q.N, status, st)
                               : launch_gemm_q8_tc(q, x, bias, residual, epi, y, yp, R, q.N, status, st, split_k);
    };
    auto split = [&](const float* x, const Planes& out, size_t n) { return out.scale != 0.0f ? launch_split_f16(x, out, n, st) : launch_split_planes(x, out, n, st); };
    FC_CUDA(cudaMemsetAsync(m->err_d, 0, sizeof(int), st));
    FC_TRY(launch_embed_rows(m->tok, m->pos, ids, pos, R, win.T, m->x, m->err_d, st));
    // model.rs:58-68: with the statistics switched on, every layer's output is summarised as it appears
    m->stats_n = 0;
    auto layer_stats = [&]() -> int {
        if (!m->stats_on) return FC_OK;
        return launch_layer_stats(m->x, Planes(), (size_t)R * d, m->stats_scratch, m->stats_d + m->stats_n++, st);
    };
    FC_TRY(layer_stats());
    for (int l = 0; l < c.n_layer; ++l) {
        const LayerDev& L = m->layers[l];
        m->pn.scale = f16 ? L.f16.n1 : 0.0f;
        m->pqkv.scale = f16 ? L.f16.heads : 0.0f;
        m->patt.scale = f16 ? L.f16.att : 0.0f;
        m->phid.scale = f16 ? L.f16.hid : 0.0f;
        FC_TRY(launch_layernorm_planes(m->x, L.ln1g, L.ln1b, nullptr, R, d, m->pn, st));
        if (tc_attn && !f32_qkv) {
            FC_TRY(product(L.qkv, L.f16.qkv, m->pn, L.qkv_b, nullptr, EPI_NONE, nullptr, &m->pqkv));
        } else {
            FC_TRY(product(L.qkv, L.f16.qkv, m->pn, L.qkv_b, nullptr, EPI_NONE, m->qkv, nullptr));
            FC_TRY(on_qkv(l));
            if (tc_attn) FC_TRY(split(m->qkv, m->pqkv, (size_t)R * 3 * d));
        }
        if (tc_attn) {
            FC_TRY(launch_attn_prefill_tc(m->pqkv, win, R, d, c.n_head, m->patt, status, st));
        } else {
            FC_TRY(launch_attn_prefill(m->qkv, win, d, c.n_head, m->att, st));
            FC_TRY(split(m->att, m->patt, (size_t)R * d));
        }
        FC_TRY(product(L.out, L.f16.out, m->patt, L.out_b, m->x, EPI_NONE, m->x, nullptr));
        m->pn.scale = f16 ? L.f16.n2 : 0.0f;
        FC_TRY(launch_layernorm_planes(m->x, L.ln2g, L.ln2b, nullptr, R, d, m->pn, st));
        FC_TRY(product(L.up, L.f16.up, m->pn, L.up_b, nullptr, EPI_GELU, nullptr, &m->phid));
        FC_TRY(product(L.down, L.f16.down, m->phid, L.down_b, m->x, EPI_NONE, m->x, nullptr));
        FC_TRY(layer_stats());
    }
    return FC_OK;
}
// The forward of a scoring batch: blocks, final LayerNorm, head and scoring tail for the scored rows.
static int score_device(fc_model* m, const ScoreSlot& s, const Windows& win, int R) {
    const fc_config& c = m->cfg;
    const int d = c.d_model, n = s.picked;
    const int *ids = (const int*)s.in_d, *pos = ids + R, *pick = pos + R + win.B + 1, *targets = pick + n;
    FC_TRY(forward_blocks_with(m, win, R, ids, pos, model_planes(m), s.status_d(), false, false, [](int) { return FC_OK; }));
    const bool f16 = m->f16 && m->lnf_scale != 0.0f;
    m->pn.n = model_planes(m);
    m->pn.scale = 0.0f;
    if (m->stats_on) {
        FC_TRY(launch_layernorm_planes(m->x, m->lnfg, m->lnfb, nullptr, R, d, m->pn, m->st));
        FC_TRY(launch_layer_stats(nullptr, m->pn, (size_t)R * d, m->stats_scratch, m->stats_d + m->stats_n++, m->st));
    }
    if (n == 0) return FC_OK;               // the forward was for its statistics
    // the head's epilogue keeps (max, sum of exponentials, first argmax) per row and 128-column tile and the
    // target's logit: [rows][V] logits never reach memory (scoring.rs:175-181 needs one number per row)
    if (f16) m->pn.scale = m->lnf_scale;
    FC_TRY(launch_layernorm_planes(m->x, m->lnfg, m->lnfb, n == R ? nullptr : pick, n, d, m->pn, m->st));
    if (f16) FC_TRY(launch_gemm_f16_score(m->head_f16, m->pn, targets, m->head_stats, m->head_tlogit, n, s.status_d(), m->st));
    else FC_TRY(launch_gemm_q8_tc_score(m->head, m->pn, targets, m->head_stats, m->head_tlogit, n, s.status_d(), m->st));
    return launch_score_combine(m->head_stats, m->head_tlogit, targets, n, (c.vocab + 127) / 128, c.vocab, s.lp_d(), s.gr_d(), m->st);
}

}  // namespace fc

// =====================================================================================
//                                      C ABI
// =====================================================================================
extern "C" {

const char* fc_last_error(void) { return fc::g_err; }

int fc_device_count(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) { cudaGetLastError(); return 0; }
    int ok = 0;
    for (int i = 0; i < n; ++i) {
        int major = 0;
        if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, i) == cudaSuccess && major == 10) ++ok;
    }
    return ok;
}

int64_t fc_take_launch_count(void) {
    const int64_t n = g_launches;
    g_launches = 0;
    return n;
}

// ------------------------------------------------------------------ standalone linear
int fc_qweight_upload(int device, const void* wq, int N, int K, fc_qweight** out) {
    if (!out) return fail(FC_E_ARG, "fc_qweight_upload: out is null");
    *out = nullptr;
    FC_TRY(select_device(device));
    fc_qweight* w = new fc_qweight;
    w->device = device;
    int rc = scratch_retain(device);
    if (rc != FC_OK) { delete w; return rc; }
    rc = w->status.create();
    if (rc == FC_OK) rc = upload_q8(w->arena, wq, N, K, &w->w, 0);
    if (rc != FC_OK) { fc_qweight_free(w); return rc; }
    *out = w;
    return FC_OK;
}

void fc_qweight_free(fc_qweight* w) {
    if (!w) return;
    cudaSetDevice(w->device);
    cudaDeviceSynchronize();
    w->arena.release();
    w->status.destroy();
    scratch_release(w->device);
    delete w;
}

int fc_q8_0_linear_dev(const fc_qweight* w, const float* x_dev, const float* bias_dev, float* y_dev,
                       int M, int math_mode, void* cuda_stream) {
    if (!w || !x_dev || !y_dev) return fail(FC_E_ARG, "fc_q8_0_linear_dev: null argument");
    if (!aligned16(x_dev) || !aligned16(y_dev) || !aligned16(bias_dev))
        return fail(FC_E_ARG, "fc_q8_0_linear_dev: x_dev, y_dev and bias_dev must be 16-byte aligned");
    if (M < 0) return fail(FC_E_SHAPE, "fc_q8_0_linear_dev: M = %d", M);
    if (M == 0) return FC_OK;
    if (math_mode != FC_MATH_FP32 && math_mode != FC_MATH_BF16X3) return fail(FC_E_ARG, "unknown math_mode %d", math_mode);
    // asking is cheaper than setting, and nearly every call finds its device current
    int current = -1;
    FC_CUDA(cudaGetDevice(&current));
    if (current != w->device) FC_CUDA(cudaSetDevice(w->device));
    cudaStream_t st = (cudaStream_t)cuda_stream;
    const GemvPart part = {w->w.qu, w->w.d, nullptr, bias_dev, y_dev, w->w.N};
    if (M == 1) return launch_gemv_alone(part, w->w.K, x_dev, st);
    if (few_rows(w->w.N, w->w.K, M)) return launch_rows_alone(part, w->w.K, x_dev, M, st);
    FC_TRY(const_cast<fc_qweight*>(w)->status.check("an earlier call on this weight"));
    const int planes = math_mode == FC_MATH_BF16X3 && w->w.K % 64 == 0 ? 2 : 3;
    const size_t n = (size_t)M * w->w.K;
    CallScratch scratch;
    Planes x;
    const size_t nw = (size_t)w->w.N * w->w.K;
    // (no more scratch than the pool keeps: with more, every call would take memory from the driver)
    if (planes == 2 && w->w.f16_exact && f16_rows(w->w.K, M) && 4 * (n + nw + M) <= kScratchKept) {
        // both operands as f16 planes, and the rows' scales behind them
        FC_TRY(scratch.take(w->device, 4 * (n + nw + M), st));
        if (scratch.p) {
            __half* p = (__half*)scratch.p;
            const F16Mat wp = {p, p + nw, w->w.N, w->w.K};
            p += 2 * nw;
            x.p[0] = p; x.p[1] = p + n; x.n = 2; x.scale = 1.0f;
            float* row_inv = (float*)(p + 2 * n);
            FC_TRY(launch_f16_planes(x_dev, M, w->w.K, x, row_inv, w->w, wp, nullptr, st));
            return launch_gemm_f16(wp, x, row_inv, bias_dev, nullptr, EPI_NONE, y_dev, nullptr, M, w->w.N, w->status.dev, st);
        }
    }
    FC_TRY(take_planes(scratch, x, planes, n, w->device, st));
    if (!scratch.p) return launch_rows_alone(part, w->w.K, x_dev, M, st);   // no memory for the planes
    FC_TRY(launch_split_planes(x_dev, x, n, st));
    return launch_gemm_q8_tc(w->w, x, bias_dev, nullptr, EPI_NONE, y_dev, nullptr, M, w->w.N, w->status.dev, st);
}

int fc_q8_0_linear(int device, const float* x, const void* wq, const float* bias, float* y,
                   int M, int K, int N, int math_mode) {
    if (!x || !wq || !y) return fail(FC_E_ARG, "fc_q8_0_linear: null argument");
    if (M < 0 || N <= 0 || K <= 0) return fail(FC_E_SHAPE, "fc_q8_0_linear: bad shape M=%d K=%d N=%d", M, K, N);
    fc_qweight* w = nullptr;
    FC_TRY(fc_qweight_upload(device, wq, N, K, &w));
    int rc = FC_OK;
    float *xd = nullptr, *bd = nullptr, *yd = nullptr;
    if (M > 0) {
        Arena tmp;
        rc = tmp.alloc_n(&xd, (size_t)M * K);
        if (rc == FC_OK) rc = tmp.alloc_n(&yd, (size_t)M * N);
        if (rc == FC_OK && bias) rc = tmp.alloc_n(&bd, (size_t)N);
        auto copy = [&](void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
            if (rc == FC_OK && cudaMemcpy(dst, src, bytes, kind) != cudaSuccess) rc = fail(FC_E_CUDA, "fc_q8_0_linear: copy failed");
        };
        copy(xd, x, (size_t)M * K * 4, cudaMemcpyHostToDevice);
        if (bias) copy(bd, bias, (size_t)N * 4, cudaMemcpyHostToDevice);
        if (rc == FC_OK) rc = fc_q8_0_linear_dev(w, xd, bd, yd, M, math_mode, nullptr);
        if (rc == FC_OK && cudaDeviceSynchronize() != cudaSuccess) rc = cuda_fail(cudaGetLastError(), "fc_q8_0_linear kernel", __FILE__, __LINE__);
        if (rc == FC_OK) rc = w->status.check("fc_q8_0_linear");
        copy(y, yd, (size_t)M * N * 4, cudaMemcpyDeviceToHost);
        tmp.release();
    }
    fc_qweight_free(w);
    return rc;
}

// ------------------------------------------------------------------------------ model
static int model_build(fc_model* m, const fc_weights* w) {
    const fc_config& c = m->cfg;
    const int d = c.d_model, F = c.d_ff, V = c.vocab;
    cudaStream_t st = m->st;
    Arena& a = m->arena;
    FC_TRY(upload_q8(a, w->token_embd_q8, V, d, &m->tok, st));
    if (c.tied) m->head = m->tok;   // loader/gpt2.rs:228-233
    else FC_TRY(upload_q8(a, w->output_q8, V, d, &m->head, st));
    FC_TRY(upload_f32(a, w->position_embd, (size_t)c.ctx * d, &m->pos, st));
    FC_TRY(upload_f32(a, w->out_norm_g, d, &m->lnfg, st));
    FC_TRY(upload_f32(a, w->out_norm_b, d, &m->lnfb, st));
    if (!w->layers) return fail(FC_E_FORMAT, "fc_weights.layers is null");
    m->layers.resize(c.n_layer);
    for (int l = 0; l < c.n_layer; ++l) {
        const fc_layer_weights& s = w->layers[l];
        LayerDev& L = m->layers[l];
        FC_TRY(upload_q8(a, s.attn_qkv_q8, 3 * d, d, &L.qkv, st));
        FC_TRY(upload_q8(a, s.attn_out_q8, d, d, &L.out, st));
        FC_TRY(upload_q8(a, s.ffn_up_q8, F, d, &L.up, st));
        FC_TRY(upload_q8(a, s.ffn_down_q8, d, F, &L.down, st));
        FC_TRY(upload_f32(a, s.attn_qkv_b, 3 * (size_t)d, &L.qkv_b, st));
        FC_TRY(upload_f32(a, s.attn_out_b, d, &L.out_b, st));
        FC_TRY(upload_f32(a, s.ffn_up_b, F, &L.up_b, st));
        FC_TRY(upload_f32(a, s.ffn_down_b, d, &L.down_b, st));
        FC_TRY(upload_f32(a, s.ln1_g, d, &L.ln1g, st));
        FC_TRY(upload_f32(a, s.ln1_b, d, &L.ln1b, st));
        FC_TRY(upload_f32(a, s.ln2_g, d, &L.ln2g, st));
        FC_TRY(upload_f32(a, s.ln2_b, d, &L.ln2b, st));
    }
    if (mega_supported(c)) {
        int full = 0;
        FC_TRY(mega_max_grid(&full));
        // One parameter table per grid size: the full GPU for a single stream, and halves,
        // quarters and eighths of it for streams decoded side by side (fc_decode_batch).
        // Per block: the four LayerNorm vectors back to back, and for every CTA of the
        // persistent kernel the slices of the four bias vectors that belong to its rows.
        std::vector<float*> lnpacks(c.n_layer, nullptr);
        std::vector<float> ln((size_t)4 * d);
        for (int l = 0; l < c.n_layer; ++l) {
            const fc_layer_weights& s = w->layers[l];
            std::copy(s.ln1_g, s.ln1_g + d, ln.begin());
            std::copy(s.ln1_b, s.ln1_b + d, ln.begin() + d);
            std::copy(s.ln2_g, s.ln2_g + d, ln.begin() + 2 * d);
            std::copy(s.ln2_b, s.ln2_b + d, ln.begin() + 3 * d);
            FC_TRY(upload_f32(a, ln.data(), ln.size(), &lnpacks[l], st));
            FC_CUDA(cudaStreamSynchronize(st));   // ln is reused by the next block
        }
        std::fill(ln.begin(), ln.end(), 0.0f);
        std::copy(w->out_norm_g, w->out_norm_g + d, ln.begin());
        std::copy(w->out_norm_b, w->out_norm_b + d, ln.begin() + d);
        FC_TRY(upload_f32(a, ln.data(), ln.size(), &m->mega_lnf, st));
        FC_CUDA(cudaStreamSynchronize(st));
        {   // the persistent kernel reads the LM head from a tile-major copy (integer tensor cores)
            unsigned char* t = nullptr;
            FC_TRY(a.alloc_n(&t, (size_t)(m->head.N_pad / kMegaStripRows) * mega_strip_bytes(m->head.K)));
            FC_TRY(launch_repack_tiles(m->head, t, st));
            m->mega_head.t = t; m->mega_head.N = m->head.N; m->mega_head.K = m->head.K;
        }
        for (int div = 1; div <= 8; div *= 2) {
            const int grid = full / div;
            if (grid < c.n_head) break;
            // the head slice and the bias slices of one CTA must fit its shared-memory buffers
            int pack = 0;
            for (int cta = 0; cta < grid; ++cta) {
                int off[4];
                pack = std::max(pack, mega_bias_offsets(d, F, cta, grid, off));
            }
            pack = (pack + 3) & ~3;
            if ((c.vocab + grid - 1) / grid + 16 > mega_head_rows_max() || pack > kMegaBiasPackMax) break;
            std::vector<MegaLayer> tab(c.n_layer);
            std::vector<float> bp((size_t)grid * pack);
            for (int l = 0; l < c.n_layer; ++l) {
                const fc_layer_weights& s = w->layers[l];
                const LayerDev& L = m->layers[l];
                std::fill(bp.begin(), bp.end(), 0.0f);
                const float* src[4] = {s.attn_qkv_b, s.attn_out_b, s.ffn_up_b, s.ffn_down_b};
                const int N[4] = {3 * d, d, F, d}, K[4] = {d, d, d, F};
                for (int cta = 0; cta < grid; ++cta) {
                    int off[4];
                    mega_bias_offsets(d, F, cta, grid, off);
                    for (int i = 0; i < 4; ++i) {
                        int r0, r1;
                        mega_cta_rows(N[i], K[i], cta, grid, &r0, &r1);
                        std::copy(src[i] + r0, src[i] + r1, bp.begin() + (size_t)cta * pack + off[i]);
                    }
                }
                float* bpd = nullptr;
                FC_TRY(upload_f32(a, bp.data(), bp.size(), &bpd, st));
                FC_CUDA(cudaStreamSynchronize(st));   // bp is reused by the next block
                tab[l] = MegaLayer{L.qkv, L.out, L.up, L.down, lnpacks[l], bpd};
            }
            MegaTable t;
            t.grid = grid;
            t.bias_pack = pack;
            FC_TRY(a.alloc_n(&t.layers, (size_t)c.n_layer));
            FC_CUDA(cudaMemcpyAsync(t.layers, tab.data(), tab.size() * sizeof(MegaLayer), cudaMemcpyHostToDevice, st));
            FC_CUDA(cudaStreamSynchronize(st));
            m->mega_tables.push_back(t);
        }
        if (!m->mega_tables.empty()) m->mega_grid = m->mega_tables[0].grid;
    }
    if (model_planes(m) == 2) FC_TRY(build_f16(m, w));            // last: out of what the model's own tables leave
    FC_CUDA(cudaStreamSynchronize(st));
    return FC_OK;
}

int fc_model_create(const fc_config* cfg, const fc_weights* w, int device, fc_model** out) {
    if (!cfg || !w || !out) return fail(FC_E_ARG, "fc_model_create: null argument");
    *out = nullptr;
    const fc_config& c = *cfg;
    if (c.n_layer <= 0 || c.d_model <= 0 || c.n_head <= 0 || c.d_ff <= 0 || c.ctx <= 0 || c.vocab <= 0)
        return fail(FC_E_SHAPE, "fc_model_create: every dimension must be positive");
    if (c.d_model % c.n_head) return fail(FC_E_DIM, "embedding_dim %d is not divisible by num_heads %d", c.d_model, c.n_head);
    if (c.d_model % 32 || c.d_ff % 32) return fail(FC_E_FORMAT, "d_model %d and d_ff %d must be multiples of 32 for Q8_0 storage", c.d_model, c.d_ff);
    const int hd = c.d_model / c.n_head;
    if (hd != 32 && hd != 64) return fail(FC_E_SHAPE, "head_dim %d is not supported (32 or 64)", hd);
    if (c.math_mode != FC_MATH_FP32 && c.math_mode != FC_MATH_BF16X3) return fail(FC_E_ARG, "unknown math_mode %d", c.math_mode);
    if (!c.tied && !w->output_q8) return fail(FC_E_FORMAT, "untied model without output.weight");
    FC_TRY(select_device(device));
    fc_model* m = new fc_model;
    m->cfg = c;
    m->device = device;
    int rc = FC_OK;
    if (cudaStreamCreateWithFlags(&m->st, cudaStreamNonBlocking) != cudaSuccess) rc = fail(FC_E_CUDA, "stream creation failed");
    if (rc == FC_OK && (cudaEventCreate(&m->ev0) != cudaSuccess || cudaEventCreate(&m->ev1) != cudaSuccess)) rc = fail(FC_E_CUDA, "event creation failed");
    if (rc == FC_OK) rc = model_build(m, w);
    if (rc == FC_OK) {
        const char* tr = getenv("FERRUM_CUDA_TRACE");
        if (tr && tr[0] == '1') rc = fc_model_set_layer_stats(m, 1);
    }
    if (rc != FC_OK) { fc_model_free(m); return rc; }
    *out = m;
    return FC_OK;
}

void fc_model_free(fc_model* m) {
    if (!m) return;
    cudaSetDevice(m->device);
    if (m->st) cudaStreamSynchronize(m->st);
    for (fc_stream* s : m->pool) fc_stream_free(s);
    m->pool.clear();
    m->arena.release();
    m->ws_arena.release();
    m->f16_arena.release();
    for (ScoreSlot& s : m->slot) s.release();
    if (m->batch.graph) cudaGraphExecDestroy(m->batch.graph);
    if (m->batch.graph4) cudaGraphExecDestroy(m->batch.graph4);
    for (cudaStream_t t : m->batch.side) cudaStreamDestroy(t);
    for (cudaEvent_t e : m->batch.side_done) cudaEventDestroy(e);
    if (m->batch.fork) cudaEventDestroy(m->batch.fork);
    m->batch.arena.release();
    m->batch.frag_arena.release();
    if (m->ev0) cudaEventDestroy(m->ev0);
    if (m->ev1) cudaEventDestroy(m->ev1);
    if (m->ev_prime) cudaEventDestroy(m->ev_prime);
    if (m->st) cudaStreamDestroy(m->st);
    delete m;
}

int fc_model_config(const fc_model* m, fc_config* out) {
    if (!m || !out) return fail(FC_E_ARG, "fc_model_config: null argument");
    *out = m->cfg;
    return FC_OK;
}

float fc_last_score_ms(const fc_model* m) { return m ? m->last_score_ms : 0.0f; }

int fc_model_set_layer_stats(fc_model* m, int on) {
    if (!m) return fail(FC_E_ARG, "fc_model_set_layer_stats: null model");
    FC_CUDA(cudaSetDevice(m->device));
    if (on && !m->stats_d) {
        FC_TRY(m->arena.alloc_n(&m->stats_d, (size_t)m->cfg.n_layer + 2));
        FC_TRY(m->arena.alloc(&m->stats_scratch, layer_stats_scratch_bytes()));
    }
    m->stats_on = on != 0;
    m->stats_n = 0;
    return FC_OK;
}

int fc_model_read_layer_stats(fc_model* m, fc_layer_stats* out, int cap) {
    if (!m || (cap > 0 && !out) || cap < 0) return fail(FC_E_ARG, "fc_model_read_layer_stats: bad argument");
    if (!m->stats_d || m->stats_n == 0) return 0;
    FC_CUDA(cudaSetDevice(m->device));
    FC_CUDA(cudaStreamSynchronize(m->st));
    std::vector<LayerStatsDev> h(m->stats_n);
    FC_CUDA(cudaMemcpy(h.data(), m->stats_d, h.size() * sizeof(LayerStatsDev), cudaMemcpyDeviceToHost));
    const int n = std::min(cap, m->stats_n);
    for (int i = 0; i < n; ++i) {
        out[i].min = h[i].min; out[i].max = h[i].max; out[i].mean = h[i].mean;
        out[i].nan_count = h[i].nan_count; out[i].inf_count = h[i].inf_count; out[i].n_elements = h[i].n;
    }
    return n;
}

// ---------------------------------------------------------------------------- scoring
// Runs B windows x T rows through the model; double log-probs / flags stay on the device
// until copied into the caller's arrays.
static int check_tc_status(fc_model* m, const char* what) {
    int status = 0;
    FC_CUDA(cudaMemcpyAsync(&status, m->tc_status, sizeof(int), cudaMemcpyDeviceToHost, m->st));
    FC_CUDA(cudaStreamSynchronize(m->st));
    if (status == 0) return FC_OK;
    cudaMemsetAsync(m->tc_status, 0, sizeof(int), m->st);
    return fail(FC_E_TIMEOUT, "a bounded wait inside a tensor-core kernel of %s ran out (status %d)", what, status);
}
// A batch of windows as the host builds it: the rows of all windows one after the other, without padding.
struct ScoreBatch {
    std::vector<int32_t> ids, pos, starts, pick, targets;
    int longest = 0;
    void clear() { ids.clear(); pos.clear(); starts.assign(1, 0); pick.clear(); targets.clear(); longest = 0; }
    // n rows; returns the first row
    int window(const int32_t* src, int n) {
        const int at = (int)ids.size();
        ids.insert(ids.end(), src, src + n);
        for (int t = 0; t < n; ++t) pos.push_back(t);
        starts.push_back(at + n);
        longest = std::max(longest, n);
        return at;
    }
    void score(int row, int32_t target) { pick.push_back(row); targets.push_back(target); }
};

static int score_issue(fc_model* m, ScoreSlot& s, const ScoreBatch& b) {
    const fc_config& c = m->cfg;
    const size_t R = b.ids.size(), n = b.pick.size(), B = b.starts.size() - 1;
    if (b.longest > c.ctx) return fail(FC_E_DIM, "Sequence length %d exceeds max_seq_len %d", b.longest, c.ctx);
    if (R > (size_t)1 << 24) return fail(FC_E_SHAPE, "too many rows in one forward: %zu", R);
    FC_TRY(check_ids(m, b.ids.data(), R));
    FC_CUDA(cudaSetDevice(m->device));
    FC_TRY(ensure_workspace(m, (int)R, model_planes(m)));
    const size_t in_bytes = 4 * (2 * R + B + 1 + 2 * n);
    s.picked = (int)n;
    FC_TRY(s.reserve(in_bytes, s.out_bytes()));
    char* at = s.in_h;
    for (const std::vector<int32_t>* v : {&b.ids, &b.pos, &b.starts, &b.pick, &b.targets}) {
        std::memcpy(at, v->data(), v->size() * 4);
        at += v->size() * 4;
    }
    cudaStream_t st = m->st;
    FC_CUDA(cudaMemcpyAsync(s.in_d, s.in_h, in_bytes, cudaMemcpyHostToDevice, st));
    FC_CUDA(cudaMemsetAsync(s.out_d, 0, 8, st));
    Windows win;
    win.B = (int)B; win.T = b.longest; win.starts = (const int*)s.in_d + 2 * R;
    FC_CUDA(cudaEventRecord(s.ev0, st));
    if (n > 0 || m->stats_on) FC_TRY(score_device(m, s, win, (int)R));
    FC_CUDA(cudaEventRecord(s.ev1, st));
    FC_CUDA(cudaMemcpyAsync(s.out_h, s.out_d, s.out_bytes(), cudaMemcpyDeviceToHost, st));
    FC_CUDA(cudaEventRecord(s.done, st));
    return FC_OK;
}

static int score_harvest(fc_model* m, ScoreSlot& s) {
    FC_CUDA(cudaEventSynchronize(s.done));
    const int status = *(const int*)s.out_h;
    if (status != 0) return fail(FC_E_TIMEOUT, "a bounded wait inside a scoring kernel ran out (status %d)", status);
    float ms = 0.0f;
    FC_CUDA(cudaEventElapsedTime(&ms, s.ev0, s.ev1));
    m->last_score_ms += ms;
    return FC_OK;
}

int fc_score_windows(fc_model* m, const int32_t* ids, const int32_t* targets, int B, int T,
                     float* logprob, uint8_t* is_greedy) {
    if (!m || !ids || !targets || !logprob || !is_greedy) return fail(FC_E_ARG, "fc_score_windows: null argument");
    if (B <= 0 || T <= 0) return fail(FC_E_SHAPE, "scoring needs B > 0 and T > 0 (got %d, %d)", B, T);
    if (T > m->cfg.ctx) return fail(FC_E_DIM, "Sequence length %d exceeds max_seq_len %d", T, m->cfg.ctx);
    if ((int64_t)B * T > (int64_t)1 << 24) return fail(FC_E_SHAPE, "too many rows in one forward: %lld", (long long)B * T);
    m->last_score_ms = 0.0f;
    ScoreBatch b;
    b.clear();
    for (int i = 0; i < B; ++i) b.window(ids + (size_t)i * T, T);
    for (int r = 0; r < B * T; ++r)
        if (targets[r] >= 0 && targets[r] < m->cfg.vocab) b.score(r, targets[r]);
    ScoreSlot& s = m->slot[0];
    FC_TRY(score_issue(m, s, b));
    FC_TRY(score_harvest(m, s));
    std::fill(logprob, logprob + (size_t)B * T, 0.0f);
    std::fill(is_greedy, is_greedy + (size_t)B * T, (uint8_t)0);
    for (int i = 0; i < s.picked; ++i) { logprob[b.pick[i]] = (float)s.lp_h()[i]; is_greedy[b.pick[i]] = s.gr_h()[i]; }
    return FC_OK;
}

}  // extern "C"

namespace {
// One window of the plan of scoring.rs:164-172.
struct Window { int seq, start, first, end; };

// (start, first target, end target exclusive) for targets from..n of one sequence.
void plan_windows(int seq, int n, int from, int T, std::vector<Window>* out) {
    const int half = std::max(1, T / 2);
    int next = std::max(from, 1);
    while (next < n) {
        const int start = next <= T ? 0 : next - half;
        const int end = std::min(start + T + 1, n);
        out->push_back(Window{seq, start, next, end});
        next = end;
    }
}

// Scores every window of `plan` in batches; seq_ids(s) gives the ids of sequence s, seq_len(s) its length. For each scored
// target calls add(seq, target, logprob, greedy), in the order of the plan. The windows of a batch lie one after the other
// without the reference's padding (scoring.rs:184-193 pads with id 0; under the causal mask no scored row sees a pad), and only
// the rows that predict a target meet the head. A batch is harvested when the next one has been queued.
template <class Ids, class Len, class Add>
int run_plan_ragged(fc_model* m, const std::vector<Window>& plan, int batch, Ids seq_ids, Len seq_len, Add add) {
    const int T = m->cfg.ctx;
    ScoreBatch b;
    auto harvest = [&](size_t w0, ScoreSlot& s) -> int {
        FC_TRY(score_harvest(m, s));
        const double* lp = s.lp_h();
        const uint8_t* gr = s.gr_h();
        for (size_t w = w0; w < std::min(w0 + batch, plan.size()); ++w)
            for (int t = plan[w].first; t < plan[w].end; ++t) add(plan[w].seq, t, *lp++, *gr++);
        return FC_OK;
    };
    int rc = FC_OK;
    size_t w0 = 0, waiting = plan.size();            // first window of the batch that is under way
    for (int k = 0; w0 < plan.size() && rc == FC_OK; w0 += batch, k ^= 1) {
        b.clear();
        for (size_t i = w0; i < std::min(w0 + batch, plan.size()); ++i) {
            const Window& w = plan[i];
            const int32_t* src = seq_ids(w.seq);
            const int at = b.window(src + w.start, std::min(w.start + T, seq_len(w.seq)) - w.start);
            for (int t = w.first; t < w.end; ++t) b.score(at + t - 1 - w.start, src[t]);
        }
        rc = score_issue(m, m->slot[k], b);
        if (rc == FC_OK && waiting < plan.size()) rc = harvest(waiting, m->slot[k ^ 1]);
        waiting = w0;
        if (rc == FC_OK && w0 + batch >= plan.size()) rc = harvest(w0, m->slot[k]);
    }
    if (rc != FC_OK) cudaStreamSynchronize(m->st);   // nothing of this call stays under way
    return rc;
}
template <class Ids, class Add>
int run_plan(fc_model* m, const std::vector<Window>& plan, int batch, Ids seq_ids, int n, Add add) {
    return run_plan_ragged(m, plan, batch, seq_ids, [n](int) { return n; }, add);
}
}  // namespace

extern "C" {

int fc_score_requests(fc_model* m, const int32_t* ids, const int64_t* offsets, const int32_t* from, int n_req, int batch_windows,
                      fc_score* scores) {
    if (!m || !scores || (n_req > 0 && (!ids || !offsets || !from))) return fail(FC_E_ARG, "fc_score_requests: null argument");
    if (n_req < 0) return fail(FC_E_SHAPE, "fc_score_requests: n_req = %d", n_req);
    m->last_score_ms = 0.0f;
    std::vector<Window> plan;
    for (int r = 0; r < n_req; ++r) {
        scores[r].logprob = 0.0; scores[r].n_tokens = 0; scores[r].greedy = 1;
        const int64_t n = offsets[r + 1] - offsets[r];
        if (n < 0 || n > (1 << 30) || from[r] < 0) return fail(FC_E_SHAPE, "fc_score_requests: request %d has length %lld, from %d", r, (long long)n, from[r]);
        FC_TRY(check_ids(m, ids + offsets[r], (size_t)n));
        plan_windows(r, (int)n, from[r], m->cfg.ctx, &plan);
    }
    if (plan.empty()) return FC_OK;
    // windows of similar length share a forward: the rows a batch pads are wasted work
    auto wlen = [&](const Window& w) { return std::min<int64_t>(w.start + m->cfg.ctx, offsets[w.seq + 1] - offsets[w.seq]) - w.start; };
    std::stable_sort(plan.begin(), plan.end(), [&](const Window& a, const Window& b) { return wlen(a) > wlen(b); });
    if (batch_windows <= 0) batch_windows = 32;
    return run_plan_ragged(m, plan, batch_windows, [&](int r) { return ids + offsets[r]; },
                           [&](int r) { return (int)(offsets[r + 1] - offsets[r]); },
                           [&](int r, int, double l, uint8_t g) { scores[r].logprob += l; scores[r].n_tokens += 1; scores[r].greedy &= (int32_t)g; });
}

int fc_token_logprobs(fc_model* m, const int32_t* ids, int n, int from, fc_score* score, float* lp, uint8_t* is_greedy) {
    if (!m || !score || (n > 0 && !ids)) return fail(FC_E_ARG, "fc_token_logprobs: null argument");
    score->logprob = 0.0; score->n_tokens = 0; score->greedy = 1;
    m->last_score_ms = 0.0f;
    if (n <= 0) return FC_OK;
    FC_TRY(check_ids(m, ids, (size_t)n));
    std::vector<Window> plan;
    plan_windows(0, n, from, m->cfg.ctx, &plan);
    // SCORE_BATCH = 32 windows per forward (scoring.rs:45)
    return run_plan(m, plan, 32, [&](int) { return ids; }, n, [&](int, int t, double l, uint8_t g) {
        score->logprob += l; score->n_tokens += 1; score->greedy &= (int32_t)g;
        if (lp) lp[t] = (float)l;
        if (is_greedy) is_greedy[t] = g;
    });
}

int fc_score_sequences(fc_model* m, const int32_t* ids, int n_seq, int seq_len, int batch_windows,
                       fc_score* scores, float* lp) {
    if (!m || !ids || !scores) return fail(FC_E_ARG, "fc_score_sequences: null argument");
    if (n_seq < 0 || seq_len < 0) return fail(FC_E_SHAPE, "fc_score_sequences: negative size");
    m->last_score_ms = 0.0f;
    for (int s = 0; s < n_seq; ++s) { scores[s].logprob = 0.0; scores[s].n_tokens = 0; scores[s].greedy = 1; }
    if (n_seq == 0 || seq_len == 0) return FC_OK;
    FC_TRY(check_ids(m, ids, (size_t)n_seq * seq_len));
    std::vector<Window> plan;
    for (int s = 0; s < n_seq; ++s) plan_windows(s, seq_len, 1, m->cfg.ctx, &plan);
    if (batch_windows <= 0) batch_windows = 32;
    if (lp) for (int s = 0; s < n_seq; ++s) lp[(size_t)s * seq_len] = 0.0f;
    return run_plan(m, plan, batch_windows, [&](int s) { return ids + (size_t)s * seq_len; }, seq_len,
                    [&](int s, int t, double l, uint8_t g) {
                        scores[s].logprob += l; scores[s].n_tokens += 1; scores[s].greedy &= (int32_t)g;
                        if (lp) lp[(size_t)s * seq_len + t] = (float)l;
                    });
}

int fc_predict_next(fc_model* m, const int32_t* ids, int n, float* probs) {
    if (!m || !ids || !probs) return fail(FC_E_ARG, "fc_predict_next: null argument");
    const fc_config& c = m->cfg;
    if (n <= 0) return fail(FC_E_SHAPE, "fc_predict_next: empty input");
    if (n > c.ctx) return fail(FC_E_DIM, "Sequence length %d exceeds max_seq_len %d", n, c.ctx);
    FC_TRY(check_ids(m, ids, (size_t)n));
    FC_CUDA(cudaSetDevice(m->device));
    FC_TRY(ensure_workspace(m, n, model_planes(m)));
    cudaStream_t st = m->st;
    FC_CUDA(cudaMemcpyAsync(m->ids_d, ids, (size_t)n * 4, cudaMemcpyHostToDevice, st));
    Windows win;
    win.B = 1; win.T = n;
    FC_TRY(forward_blocks_with(m, win, n, m->ids_d, nullptr, model_planes(m), m->tc_status, false, false, [](int) { return FC_OK; }));
    FC_TRY(launch_gemv_row(m->head, m->x + (size_t)(n - 1) * c.d_model, RowNorm{m->lnfg, m->lnfb, 1e-5f}, nullptr, nullptr, EPI_NONE, m->logits,
                           nullptr, st));
    FC_TRY(launch_softmax_row(m->logits, c.vocab, m->probs_d, st));
    FC_CUDA(cudaMemcpyAsync(probs, m->probs_d, (size_t)c.vocab * 4, cudaMemcpyDeviceToHost, st));
    return check_tc_status(m, "predict_next");
}

// ----------------------------------------------------------------------------- streams
static int stream_create(fc_model* m, fc_stream** out) {
    const fc_config& c = m->cfg;
    fc_stream* s = new fc_stream;
    s->m = m;
    Arena& a = s->arena;
    const size_t cache = (size_t)c.n_layer * c.ctx * c.d_model;
    s->queue_cap = c.ctx + 8;
    int rc = a.alloc_n(&s->kc, cache);
    if (rc == FC_OK) rc = a.alloc_n(&s->vc, cache);
    if (rc == FC_OK) rc = a.alloc_n(&s->x, (size_t)c.d_model);
    if (rc == FC_OK) rc = a.alloc_n(&s->q, (size_t)c.d_model);
    if (rc == FC_OK) rc = a.alloc_n(&s->att, (size_t)c.d_model);
    if (rc == FC_OK) rc = a.alloc_n(&s->hid, (size_t)c.d_ff);
    if (rc == FC_OK) rc = a.alloc_n(&s->logits, (size_t)c.vocab);
    if (rc == FC_OK) rc = a.alloc_n(&s->probs, (size_t)c.vocab);
    if (rc == FC_OK) rc = a.alloc_n(&s->queue, (size_t)s->queue_cap);
    if (rc == FC_OK) rc = a.alloc_n(&s->state, 1);
    if (rc == FC_OK) rc = a.alloc_n(&s->stats, kRowStats);
    if (rc == FC_OK) rc = a.alloc_n(&s->qkv, (size_t)3 * c.d_model);
    if (rc == FC_OK) rc = a.alloc_n(&s->status, 1);
    if (rc == FC_OK && cudaMemsetAsync(s->status, 0, sizeof(int), m->st) != cudaSuccess) rc = fail(FC_E_CUDA, "status word initialisation failed");
    const int hd = c.d_model / c.n_head;
    if (rc == FC_OK) rc = attn_step_split(c.n_head, hd, c.ctx, &s->attn_split, &s->split_from);
    if (rc == FC_OK && block_step_covers(c.d_model, c.n_head, c.d_ff, c.ctx, false)) {
        rc = a.alloc_n(&s->parts_a, (size_t)c.n_head * c.d_model);
        if (rc == FC_OK) rc = a.alloc_n(&s->parts_m, (size_t)block_step_slices(c.d_ff, false) * c.d_model);
        s->split_from = INT_MAX;
    }
    if (rc == FC_OK && m->mega_grid > 0) {
        s->attn_splits = std::max(1, std::min(8, m->mega_grid / c.n_head));
        rc = a.alloc_n(&s->partg, (size_t)c.n_head * s->attn_splits * (hd + 2));
        if (rc == FC_OK) rc = a.alloc_n(&s->x1g, (size_t)c.d_model);
        if (rc == FC_OK) rc = a.alloc_n(&s->statg, (size_t)m->mega_grid * 4);
        if (rc == FC_OK) rc = a.alloc_n(&s->bar, 1);
        if (rc == FC_OK) rc = a.alloc_n(&s->trace, (size_t)m->mega_grid * kTraceCap);
    }
    if (rc == FC_OK && (cudaEventCreate(&s->ev0) != cudaSuccess || cudaEventCreate(&s->ev1) != cudaSuccess)) rc = fail(FC_E_CUDA, "event creation failed");
    if (rc == FC_OK) rc = set_state(s, 0, 0, 0, -1, 0);
    if (rc == FC_OK && cudaStreamSynchronize(m->st) != cudaSuccess) rc = fail(FC_E_CUDA, "stream initialisation failed");
    if (rc != FC_OK) { fc_stream_free(s); return rc; }
    *out = s;
    return FC_OK;
}
int fc_stream_create(fc_model* m, fc_stream** out) {
    if (!m || !out) return fail(FC_E_ARG, "fc_stream_create: null argument");
    *out = nullptr;
    FC_CUDA(cudaSetDevice(m->device));
    return with_room(m, [&] { return stream_create(m, out); });
}

void fc_stream_free(fc_stream* s) {
    if (!s) return;
    cudaSetDevice(s->m->device);
    cudaStreamSynchronize(s->m->st);
    if (s->cs) { cudaStreamSynchronize(s->cs); cudaStreamDestroy(s->cs); }
    if (s->cs_done) cudaEventDestroy(s->cs_done);
    drop_graphs(s);
    if (s->ev0) cudaEventDestroy(s->ev0);
    if (s->ev1) cudaEventDestroy(s->ev1);
    s->arena.release();
    delete s;
}

int fc_stream_reset(fc_stream* s) {
    if (!s) return fail(FC_E_ARG, "fc_stream_reset: null stream");
    FC_CUDA(cudaSetDevice(s->m->device));
    s->host_pos = 0;
    return set_state(s, 0, 0, 0, -1, 0);
}

int fc_cached_len(const fc_stream* s) { return s ? s->host_pos : 0; }

int fc_stream_set_trace(fc_stream* s, int on) {
    if (!s) return fail(FC_E_ARG, "fc_stream_set_trace: null stream");
    if (on && !s->trace) return fail(FC_E_SHAPE, "tracing needs the persistent decode kernel");
    s->trace_on = on != 0;
    return FC_OK;
}

int fc_stream_read_trace(fc_stream* s, uint64_t* out, int cap) { return fc_stream_read_trace_cta(s, 0, out, cap); }

int fc_stream_read_trace_cta(fc_stream* s, int cta, uint64_t* out, int cap) {
    if (!s || !out || cap < 0) return fail(FC_E_ARG, "fc_stream_read_trace: bad argument");
    if (!s->trace) return 0;
    if (cta < 0 || cta >= s->m->mega_grid) return fail(FC_E_ARG, "fc_stream_read_trace: the kernel runs %d CTAs", s->m->mega_grid);
    FC_CUDA(cudaSetDevice(s->m->device));
    FC_CUDA(cudaStreamSynchronize(s->m->st));
    std::vector<unsigned long long> h(kTraceCap);
    FC_CUDA(cudaMemcpy(h.data(), s->trace + (size_t)cta * kTraceCap, kTraceCap * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
    int n = 0;
    while (n < kTraceCap && n < cap && h[n] != 0) { out[n] = h[n]; ++n; }
    return n;
}

int fc_stream_set_mode(fc_stream* s, int mode) {
    if (!s) return fail(FC_E_ARG, "fc_stream_set_mode: null stream");
    if (mode == FC_DECODE_PERSISTENT && s->m->mega_grid <= 0)
        return fail(FC_E_SHAPE, "the persistent decode kernel does not support this model shape");
    if (mode != FC_DECODE_PERSISTENT && mode != FC_DECODE_PER_KERNEL && mode != FC_DECODE_AUTO) return fail(FC_E_ARG, "unknown decode mode %d", mode);
    s->mode = mode;
    return FC_OK;
}
float fc_last_decode_ms(const fc_stream* s) { return s ? s->last_decode_ms : 0.0f; }

__global__ void bump_state_kernel(StepState* st, int by) {
    if (st->done | st->error) return;
    st->pos += by;
    st->fed += by;
}

// CachedTransformer::prime (slm/cached.rs:129-136) feeds the ids one at a time; on an empty
// cache the same rows come out of ONE window forward (TransformerBlock::forward,
// layer/transformer.rs:314-534, equals forward_with_cache row by row: transformer.rs:669-716),
// so the n ids in queue[0..n) of each of the S streams go through every block as S windows of
// n rows, each block's K and V rows are copied into the streams' caches, and only the
// last row of a window meets the head.
// Very short prompts stay on the token-by-token path (one persistent-kernel launch); with few
// rows the GEMMs split K over a cluster so that more SMs take part.
// Returns FC_OK with *used = 0 when the shape is not covered (the caller feeds token by token).
constexpr int kPrimeBatchMin = 8;
static int prime_batched(fc_stream* const* ss, int S, int n, int last_mode, int* used, float* const* kcs_dev = nullptr,
                         float* const* vcs_dev = nullptr) {
    fc_model* m = ss[0]->m;
    const fc_config& c = m->cfg;
    const int d = c.d_model, hd = d / c.n_head, R = S * n;
    *used = 0;
    if (R < kPrimeBatchMin || n < 2 || (hd != 32 && hd != 64)) return FC_OK;
    for (int i = 0; i < S; ++i)
        if (ss[i]->host_pos != 0) return FC_OK;
    cudaStream_t st = m->st;
    // prompts keep f32 rounding (3 planes) unless the model's scoring mode is the 2-plane one and there are many rows
    const int planes = R >= 256 && tensor_attention(m) && model_planes(m) == 2 ? 2 : 3;
    FC_TRY(ensure_workspace(m, R, planes));
    for (int i = 0; i < S; ++i)
        FC_CUDA(cudaMemcpyAsync(m->ids_d + (size_t)i * n, ss[i]->queue, (size_t)n * sizeof(int), cudaMemcpyDeviceToDevice, st));
    const size_t layer_stride = (size_t)c.ctx * d;
    // rows [q | k | v] of window i -> cache positions 0..n-1 of stream i
    auto to_caches = [&](int l) -> int {
        if (kcs_dev && vcs_dev) return launch_scatter_kv(m->qkv, kcs_dev, vcs_dev, l * layer_stride, S, n, d, st);
        for (int i = 0; i < S; ++i) {
            const float* rows = m->qkv + (size_t)i * n * 3 * d;
            FC_CUDA(cudaMemcpy2DAsync(ss[i]->kc + l * layer_stride, (size_t)d * 4, rows + d, (size_t)3 * d * 4, (size_t)d * 4, n,
                                      cudaMemcpyDeviceToDevice, st));
            FC_CUDA(cudaMemcpy2DAsync(ss[i]->vc + l * layer_stride, (size_t)d * 4, rows + 2 * d, (size_t)3 * d * 4, (size_t)d * 4, n,
                                      cudaMemcpyDeviceToDevice, st));
        }
        return FC_OK;
    };
    Windows win;
    win.B = S; win.T = n;
    // a wait that runs out: fc_decode_batch reads the model's word, read_state the stream's
    FC_TRY(forward_blocks_with(m, win, R, m->ids_d, nullptr, planes, kcs_dev ? m->tc_status : ss[0]->status, true, true, to_caches));
    *used = 1;
    for (int i = 0; i < S; ++i) {
        fc_stream* s = ss[i];
        if (last_mode == STEP_NOHEAD) {
            bump_state_kernel<<<1, 1, 0, st>>>(s->state, n);
            FC_LAUNCHED();
            continue;
        }
        // the head sees the last row only; its tail advances the position by one
        bump_state_kernel<<<1, 1, 0, st>>>(s->state, n - 1);
        FC_LAUNCHED();
        FC_TRY(launch_head(s, m->x + ((size_t)i * n + n - 1) * d, last_mode));
    }
    return FC_OK;
}

// Feeds queue[0..n) (already uploaded) from the current position; the last step runs in
// `last_mode`, the ones before it skip the head (its output would be discarded).
static int feed_queued(fc_stream* s, int n, int last_mode) {
    int used = 0;
    FC_TRY(prime_batched(&s, 1, n, last_mode, &used));
    if (used) return FC_OK;
    return run_steps(s, n, STEP_NOHEAD, last_mode, s->host_pos);
}

static int feed_ids(fc_stream* s, const int32_t* ids, int n, float* probs) {
    fc_model* m = s->m;
    const fc_config& c = m->cfg;
    FC_TRY(check_ids(m, ids, (size_t)n));
    if (s->host_pos + n > c.ctx)
        return fail(FC_E_DIM, "KvCache full (%d positions): clear and re-prime to continue", c.ctx);
    if (n == 0) return FC_OK;
    cudaStream_t st = m->st;
    FC_CUDA(cudaMemcpyAsync(s->queue, ids, (size_t)n * 4, cudaMemcpyHostToDevice, st));
    FC_TRY(set_state(s, 0, 0, n, -1, /*keep_pos=*/1));
    FC_TRY(feed_queued(s, n, probs ? STEP_PROBS : STEP_NOHEAD));
    if (probs) FC_CUDA(cudaMemcpyAsync(probs, s->probs, (size_t)c.vocab * 4, cudaMemcpyDeviceToHost, st));
    StepState hs;
    FC_TRY(read_state(s, &hs));
    if (hs.error) return fail(hs.error, "decode step rejected a token or position on the device");
    s->host_pos = hs.pos;
    return FC_OK;
}

int fc_feed(fc_stream* s, int32_t token, float* probs) {
    if (!s) return fail(FC_E_ARG, "fc_feed: null stream");
    FC_CUDA(cudaSetDevice(s->m->device));
    return feed_ids(s, &token, 1, probs);
}

int fc_prime(fc_stream* s, const int32_t* ids, int n, float* probs) {
    if (!s || (n > 0 && !ids)) return fail(FC_E_ARG, "fc_prime: null argument");
    if (n < 0) return fail(FC_E_SHAPE, "fc_prime: n = %d", n);
    FC_TRY(fc_stream_reset(s));
    return feed_ids(s, ids, n, probs);
}

int fc_generate_greedy(fc_stream* s, const int32_t* prompt, int n, int max_new, int32_t eos,
                       const volatile int32_t* cancel, int32_t* out, int* n_out) {
    if (!s || !prompt || !n_out || (max_new > 0 && !out)) return fail(FC_E_ARG, "fc_generate_greedy: null argument");
    *n_out = 0;
    if (n <= 0) return fail(FC_E_SHAPE, "fc_generate_greedy: empty prompt (pass the BOS id, token_stream.rs:84-86)");
    if (max_new < 0) return fail(FC_E_SHAPE, "fc_generate_greedy: max_new = %d", max_new);
    fc_model* m = s->m;
    const fc_config& c = m->cfg;
    FC_CUDA(cudaSetDevice(m->device));
    FC_TRY(check_ids(m, prompt, (size_t)n));
    cudaStream_t st = m->st;
    const int cap = std::max(1, (int)c.ctx), keep = std::max(1, cap / 2);
    s->last_decode_ms = 0.0f;

    // window = the last `cap` prompt ids (token_stream.rs:87-89)
    std::vector<int32_t> window(prompt + std::max(0, n - cap), prompt + n);
    int made = 0;          // tokens already copied to `out` (earlier windows)
    bool done = false, cancelled = false;
    // Starts a window: reset, upload, prime. The last prime step selects the next token when
    // one is still wanted.
    auto start_window = [&](bool select) -> int {
        FC_TRY(fc_stream_reset(s));
        FC_CUDA(cudaMemcpyAsync(s->queue, window.data(), window.size() * 4, cudaMemcpyHostToDevice, st));
        FC_TRY(set_state(s, 0, 0, (int)window.size(), eos, 0));
        return feed_queued(s, (int)window.size(), select ? STEP_SELECT : STEP_PROBS);
    };
    // Reads back what the device appended to the current window; sets `done` on eos.
    auto harvest = [&]() -> int {
        StepState hs;
        FC_TRY(read_state(s, &hs));
        if (hs.error) return fail(hs.error, "decode step rejected a token or position on the device");
        const int have = hs.tail - (int)window.size();
        if (have > 0) {
            window.resize(hs.tail);
            FC_CUDA(cudaMemcpy(window.data() + hs.tail - have, s->queue + hs.tail - have, (size_t)have * 4, cudaMemcpyDeviceToHost));
            for (int i = 0; i < have && made < max_new; ++i) out[made++] = window[hs.tail - have + i];
        }
        s->host_pos = hs.pos;
        done = hs.done != 0;
        return FC_OK;
    };

    FC_TRY(start_window(max_new > 0));
    FC_CUDA(cudaEventRecord(s->ev0, st));
    int win_start_len = (int)window.size();  // ids in the window when it was primed
    int gen_win = max_new > 0 ? 1 : 0;       // tokens selected inside this window (issued)
    // feed i (1-based) pushes generated token i; it selects token i+1 unless it is the last.
    // Consecutive selecting feeds are issued as one batch of at most 32 steps.
    int i = 1;
    while (i <= max_new && !done) {
        if (cancel && *cancel) { cancelled = true; break; }
        if (win_start_len + gen_win > cap) {
            // the window outgrew the context: keep the last cap/2 ids and re-prime
            // (token_stream.rs:162-165)
            const bool select = i < max_new;
            FC_TRY(harvest());
            if (done) break;
            window.erase(window.begin(), window.end() - keep);
            FC_TRY(start_window(select));
            win_start_len = (int)window.size();
            gen_win = select ? 1 : 0;
            i += 1;
        } else {
            // selecting feeds i..max_new-1, as many as stay inside the context
            const int k = std::min(std::min(max_new - i, 32), cap - win_start_len - gen_win + 1);
            if (k >= 1) {
                FC_TRY(decode_steps(s, k, STEP_SELECT, win_start_len + gen_win - 1));
                gen_win += k;
                i += k;
            } else {
                FC_TRY(decode_steps(s, 1, STEP_PROBS, win_start_len + gen_win - 1));   // the last feed selects nothing
                i += 1;
            }
        }
        // eos can only be noticed on the host at a synchronisation point
        if (eos >= 0) FC_TRY(harvest());
    }
    FC_CUDA(cudaEventRecord(s->ev1, st));
    FC_TRY(harvest());
    FC_CUDA(cudaEventElapsedTime(&s->last_decode_ms, s->ev0, s->ev1));
    *n_out = made;
    if (cancelled) return fail(FC_E_CANCELLED, "generation cancelled after %d tokens", made);
    return FC_OK;
}

int fc_sample_logits(int device, const float* logits, int n, const fc_sampling* params, const int32_t* recent, int n_recent,
                     uint64_t* rng_state, int32_t* token) {
    if (!logits || !params || !rng_state || !token || (n_recent > 0 && !recent)) return fail(FC_E_ARG, "fc_sample_logits: null argument");
    if (n <= 0 || n_recent < 0) return fail(FC_E_SHAPE, "fc_sample_logits: n = %d, n_recent = %d", n, n_recent);
    FC_TRY(select_device(device));
    Arena a;
    float* d_logits = nullptr;
    int* d_recent = nullptr;
    unsigned long long* d_rng = nullptr;
    int* d_tok = nullptr;
    int rc = a.alloc_n(&d_logits, (size_t)n);
    if (rc == FC_OK) rc = a.alloc_n(&d_recent, (size_t)std::max(n_recent, 1));
    if (rc == FC_OK) rc = a.alloc_n(&d_rng, 1);
    if (rc == FC_OK) rc = a.alloc_n(&d_tok, 1);
    auto copy = [&](void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
        if (rc == FC_OK && bytes && cudaMemcpy(dst, src, bytes, kind) != cudaSuccess) rc = fail(FC_E_CUDA, "fc_sample_logits: copy failed");
    };
    copy(d_logits, logits, (size_t)n * 4, cudaMemcpyHostToDevice);
    copy(d_recent, recent, (size_t)n_recent * 4, cudaMemcpyHostToDevice);
    copy(d_rng, rng_state, 8, cudaMemcpyHostToDevice);
    if (rc == FC_OK) rc = launch_sample(d_logits, n, 0, *params, d_recent, n_recent, d_rng, nullptr, 0, nullptr, d_tok, nullptr);
    if (rc == FC_OK && cudaDeviceSynchronize() != cudaSuccess) rc = fail(FC_E_CUDA, "fc_sample_logits: the sampler failed");
    copy(token, d_tok, 4, cudaMemcpyDeviceToHost);
    copy(rng_state, d_rng, 8, cudaMemcpyDeviceToHost);
    a.release();
    return rc;
}

int fc_generate_sampled(fc_stream* s, const int32_t* prompt, int n, int max_new, int32_t eos, const fc_sampling* params,
                        uint64_t* rng_state, const volatile int32_t* cancel, int32_t* out, int* n_out) {
    if (!s || !prompt || !n_out || !params || !rng_state || (max_new > 0 && !out)) return fail(FC_E_ARG, "fc_generate_sampled: null argument");
    *n_out = 0;
    if (n <= 0) return fail(FC_E_SHAPE, "fc_generate_sampled: empty prompt (pass the BOS id, token_stream.rs:84-86)");
    if (max_new < 0) return fail(FC_E_SHAPE, "fc_generate_sampled: max_new = %d", max_new);
    fc_model* m = s->m;
    const fc_config& c = m->cfg;
    FC_CUDA(cudaSetDevice(m->device));
    FC_TRY(check_ids(m, prompt, (size_t)n));
    cudaStream_t st = m->st;
    const int cap = std::max(1, (int)c.ctx), keep = std::max(1, cap / 2);
    if (!s->rng_d) FC_TRY(s->arena.alloc_n(&s->rng_d, 1));
    FC_CUDA(cudaMemcpyAsync(s->rng_d, rng_state, 8, cudaMemcpyHostToDevice, st));
    s->last_decode_ms = 0.0f;
    // window = the last `cap` prompt ids (token_stream.rs:87-89); priming leaves the distribution
    // of the next token in s->probs
    std::vector<int32_t> window(prompt + std::max(0, n - cap), prompt + n);
    auto start_window = [&]() -> int {
        FC_TRY(fc_stream_reset(s));
        FC_CUDA(cudaMemcpyAsync(s->queue, window.data(), window.size() * 4, cudaMemcpyHostToDevice, st));
        FC_TRY(set_state(s, 0, 0, (int)window.size(), eos, 0));
        return feed_queued(s, (int)window.size(), STEP_PROBS);
    };
    FC_TRY(start_window());
    FC_CUDA(cudaEventRecord(s->ev0, st));
    int made = 0;
    bool cancelled = false, timed = false;
    int rc = FC_OK;
    // A draw appends its token to the queue on the device (or raises `done` on eos, which turns what follows into no-ops) and
    // the feed reads it there, so the host reads back once per `batch` draws; with a cancel flag, which is polled before every
    // draw, that is each one. A draw that makes the window outgrow the context goes alone: its re-prime starts on the host.
    const int batch = cancel ? 1 : 16;
    auto draw = [&]() { return launch_sample(s->probs, c.vocab, 1, *params, s->queue, 0, s->rng_d, s->queue, s->queue_cap, s->state, nullptr, st); };
    auto issue = [&](int k, bool feed) -> int {
        for (int i = 1; i <= k; ++i) {
            FC_TRY(draw());
            // the feed (or re-prime) after the last requested token keeps the stream continuable, as the reference's call
            // order does, but its distribution is not used here: it stays outside the timed region
            if (made + i == max_new) { FC_CUDA(cudaEventRecord(s->ev1, st)); timed = true; }
            if (feed) FC_TRY(decode_steps(s, 1, STEP_PROBS, (int)window.size() + i - 1));   // feed(next): the distribution of the token after it
        }
        return FC_OK;
    };
    // Reads back what the draws appended to the window.
    auto harvest = [&](bool* done) -> int {
        StepState hs;
        FC_TRY(read_state(s, &hs));
        if (hs.error) return fail(hs.error, "decode step rejected a token or position on the device");
        const int have = hs.tail - (int)window.size();
        if (have > 0) {
            window.resize(hs.tail);
            FC_CUDA(cudaMemcpy(window.data() + hs.tail - have, s->queue + hs.tail - have, (size_t)have * 4, cudaMemcpyDeviceToHost));
            for (int i = 0; i < have; ++i) out[made++] = window[hs.tail - have + i];
        }
        *done = hs.done != 0;
        return FC_OK;
    };
    while (made < max_new) {
        if (cancel && *cancel) { cancelled = true; break; }
        const int k = std::min(std::min(max_new - made, batch), cap - (int)window.size());
        bool done = false;
        rc = issue(std::max(k, 1), k > 0);
        if (rc == FC_OK) rc = harvest(&done);
        if (rc != FC_OK || done) break;                       // eos: nothing was appended
        if (k <= 0) {
            // the window outgrew the context: keep the last cap/2 ids and re-prime (token_stream.rs:162-165)
            window.erase(window.begin(), window.end() - keep);
            rc = start_window();
            if (rc != FC_OK) break;
        }
    }
    if (rc == FC_OK) {
        if (!timed) FC_CUDA(cudaEventRecord(s->ev1, st));
        StepState hs;
        rc = read_state(s, &hs);
        if (rc == FC_OK && hs.error) rc = fail(hs.error, "decode step rejected a token or position on the device");
        if (rc == FC_OK) {
            s->host_pos = hs.pos;
            FC_CUDA(cudaEventElapsedTime(&s->last_decode_ms, s->ev0, s->ev1));
        }
    }
    FC_CUDA(cudaMemcpy(rng_state, s->rng_d, 8, cudaMemcpyDeviceToHost));
    if (rc != FC_OK) return rc;
    *n_out = made;
    if (cancelled) return fail(FC_E_CANCELLED, "generation cancelled after %d tokens", made);
    return FC_OK;
}

// ------------------------------------------------------------------- lock-step decode
// Fragment-major copies of every matrix, made once per model on the first batched decode.
static int batch_make_frags(fc_model* m) {
    BatchCtx& b = m->batch;
    if (b.frags) return FC_OK;
    cudaStream_t st = m->st;
    auto make = [&](const QMat& w, QFrag* out) -> int {
        void *q = nullptr, *d = nullptr;
        FC_TRY(b.frag_arena.alloc(&q, frag_quant_bytes(w)));
        FC_TRY(b.frag_arena.alloc(&d, frag_scale_bytes(w)));
        FC_TRY(launch_repack_frag(w, q, d, st));
        out->q = q; out->d = d; out->N = w.N; out->K = w.K; out->N_pad = w.N_pad;
        return FC_OK;
    };
    const int L = m->cfg.n_layer;
    b.qkv.resize(L); b.out.resize(L); b.up.resize(L); b.down.resize(L);
    int rc = FC_OK;
    for (int l = 0; l < L && rc == FC_OK; ++l) {
        rc = make(m->layers[l].qkv, &b.qkv[l]);
        if (rc == FC_OK) rc = make(m->layers[l].out, &b.out[l]);
        if (rc == FC_OK) rc = make(m->layers[l].up, &b.up[l]);
        if (rc == FC_OK) rc = make(m->layers[l].down, &b.down[l]);
    }
    if (rc == FC_OK) rc = make(m->head, &b.head);
    if (rc == FC_OK && cudaStreamSynchronize(st) != cudaSuccess) rc = fail(FC_E_CUDA, "fragment-major weight copy failed");
    if (rc != FC_OK) { b.frag_arena.release(); return rc; }
    b.frags = true;
    return FC_OK;
}

static int batch_ensure(fc_model* m, int S, int out_cap) {
    BatchCtx& b = m->batch;
    if (S <= b.cap && out_cap <= b.out_cap) return FC_OK;
    FC_CUDA(cudaStreamSynchronize(m->st));
    if (b.graph) { cudaGraphExecDestroy(b.graph); b.graph = nullptr; }
    if (b.graph4) { cudaGraphExecDestroy(b.graph4); b.graph4 = nullptr; }
    b.graph_S = 0;
    b.arena.release();
    b.cap = b.out_cap = 0;
    const fc_config& c = m->cfg;
    // two f16 columns per stream; a ragged last group reads (never uses) up to 128 columns past its own
    const size_t cap = std::max(S, b.cap), oc = std::max(out_cap, b.out_cap), C = kBatchMaxStreams * 2 + 128;
    const size_t d = c.d_model, F = c.d_ff;
    Arena& a = b.arena;
    FC_TRY(a.alloc_n(&b.x, cap * d));
    FC_TRY(a.alloc_n(&b.x2, cap * d));
    FC_TRY(a.alloc_n(&b.part, (size_t)skinny_max_splits() * cap * d));
    FC_TRY(a.alloc_n(&b.qkv_f, cap * 3 * d));
    FC_TRY(a.alloc_n(&b.logits, cap * (size_t)m->head.N_pad));
    FC_TRY(a.alloc(&b.xp, C * d * 2));
    FC_TRY(a.alloc(&b.ap, C * d * 2));
    FC_TRY(a.alloc(&b.hp, C * F * 2));
    // rows past the live streams are read by the MMA tiles: they stay zero
    FC_CUDA(cudaMemsetAsync(b.xp, 0, C * d * 2, m->st));
    FC_CUDA(cudaMemsetAsync(b.ap, 0, C * d * 2, m->st));
    FC_CUDA(cudaMemsetAsync(b.hp, 0, C * F * 2, m->st));
    FC_TRY(a.alloc_n(&b.cur, cap));
    FC_TRY(a.alloc_n(&b.done, cap));
    FC_TRY(a.alloc_n(&b.n_out, cap));
    FC_TRY(a.alloc_n(&b.out_tok, cap * std::max<size_t>(oc, 1)));
    FC_TRY(a.alloc_n(&b.pos, kBatchMaxStreams));   // one position word per group of the step graph, all equal
    FC_TRY(a.alloc_n(&b.kcs, cap));
    FC_TRY(a.alloc_n(&b.vcs, cap));
    FC_TRY(a.alloc_n(&b.queues, cap));
    FC_TRY(a.alloc_n(&b.states, cap));
    b.cap = (int)cap;
    b.out_cap = (int)oc;
    return FC_OK;
}

// The buffers of one group of streams (streams s0 .. s0 + S of a wave). Every per-stream array is indexed by the
// stream, so a group is a set of offsets into the wave's buffers, its own position word and the CUDA stream its
// kernels are issued on.
struct BatchView {
    int S;
    float *x, *x2, *part, *qkv_f, *logits;
    void *xp, *ap, *hp;
    int *cur, *done, *n_out, *out_tok, *pos;
    float **kcs, **vcs;
    cudaStream_t st;
    int max_warps;                     // per CTA of the products: fewer when several groups run side by side
    bool long_k_block;                 // the 32-warp tile of the long-K products: up to two groups
};

static BatchView batch_view(fc_model* m, int s0, int S, int group_index, cudaStream_t st, int n_groups = 1) {
    const fc_config& c = m->cfg;
    BatchCtx& b = m->batch;
    const size_t d = c.d_model, F = c.d_ff, o = (size_t)s0;
    BatchView v;
    v.S = S;
    v.x = b.x + o * d;
    v.x2 = b.x2 + o * d;
    v.part = b.part + (size_t)skinny_max_splits() * o * d;        // [splits][S][d] of the group
    v.qkv_f = b.qkv_f + o * 3 * d;
    v.logits = b.logits + o * (size_t)m->head.N_pad;
    v.xp = (char*)b.xp + 2 * o * d * 2;                           // two f16 columns per stream
    v.ap = (char*)b.ap + 2 * o * d * 2;
    v.hp = (char*)b.hp + 2 * o * F * 2;
    v.cur = b.cur + o; v.done = b.done + o; v.n_out = b.n_out + o;
    v.out_tok = b.out_tok + o * (size_t)b.out_cap;
    v.pos = b.pos + group_index;
    v.kcs = b.kcs + o; v.vcs = b.vcs + o;
    v.st = st;
    v.max_warps = n_groups > 1 ? 8 : 16;
    v.long_k_block = n_groups <= 2;
    return v;
}

// The tail of a step: final LayerNorm (model.rs:51-71 layer list: ..., LayerNorm, Linear, Softmax), head,
// greedy pick. With `part` the last down-projection is still in partial sums, which the LayerNorm adds.
static int batch_head_and_pick(fc_model* m, const BatchView& v, int eos, const float* x, const float* part, int n_part,
                               const float* part_bias, float* x_other, int advance) {
    const fc_config& c = m->cfg;
    BatchCtx& b = m->batch;
    FC_TRY(launch_ln_rows_f16(x, part, n_part, part_bias, x_other, m->lnfg, m->lnfb, v.S, c.d_model, v.xp, v.st));
    SkinnyOut out;
    out.max_warps = v.max_warps; out.long_k_block = v.long_k_block;
    out.y = v.logits; out.ldy = m->head.N_pad;
    FC_TRY(launch_skinny_q8(b.head, v.S, v.xp, nullptr, EPI_NONE, out, nullptr, v.st));
    return launch_pick_batch(v.logits, m->head.N_pad, c.vocab, v.S, eos, v.cur, v.done, v.n_out, v.out_tok, b.out_cap, v.pos, advance, v.st);
}

// One step for the S streams of a group: CachedTransformer::feed (cached.rs:100-125) on every stream's current
// token at the shared position, then the greedy pick per stream. Seven kernels per block.
//  * Up to 16 streams every kernel is a chain of a few memory round trips and nothing else: the
//    out- and down-projections add bias and residual in their own epilogue (in place).
//  * Beyond that the out- and down-projections split K over CTAs (their 1024-odd output rows
//    alone would leave most SMs idle) and leave partial sums; the LayerNorm kernel that reads the
//    residual stream next adds them, the bias and the residual in a fixed order
//    (transformer.rs:272,293).
static int batch_launch_step(fc_model* m, const BatchView& v, int eos) {
    const fc_config& c = m->cfg;
    BatchCtx& b = m->batch;
    cudaStream_t st = v.st;
    const int S = v.S, d = c.d_model, F = c.d_ff;
    const size_t layer_stride = (size_t)c.ctx * d;
    const bool split_k = S > 16;
    FC_TRY(launch_embed_batch(m->tok, m->pos, v.cur, v.pos, S, v.x, st));
    float *x = v.x, *x_other = v.x2;       // the stream as of the last completed residual add, and the other buffer
    const float* part_bias = nullptr;      // bias of the product whose partial sums are pending
    int n_part = 0;
    // LayerNorm of the residual stream, completed first when partial sums are pending
    auto normed = [&](const float* g, const float* be) -> int {
        FC_TRY(launch_ln_rows_f16(x, n_part > 0 ? v.part : nullptr, n_part, part_bias, x_other, g, be, S, d, v.xp, st));
        if (n_part > 0) std::swap(x, x_other);   // the completed stream now lives in the other buffer
        n_part = 0;
        part_bias = nullptr;
        return FC_OK;
    };
    // x <- x + (W in + bias): as partial sums for the next LayerNorm, or finished in the epilogue
    auto project_add = [&](const QFrag& w, const void* in, const float* bias) -> int {
        SkinnyOut o;
        o.max_warps = v.max_warps; o.long_k_block = v.long_k_block;
        if (split_k) {
            o.part = v.part;
            FC_TRY(launch_skinny_q8(w, S, in, nullptr, EPI_NONE, o, &n_part, st));
            part_bias = bias;
            return FC_OK;
        }
        o.y = x; o.ldy = d; o.residual = x;
        return launch_skinny_q8(w, S, in, bias, EPI_NONE, o, nullptr, st);
    };
    SkinnyOut oq, oh;
    oq.max_warps = oh.max_warps = v.max_warps;
    oq.long_k_block = oh.long_k_block = v.long_k_block;
    oq.y = v.qkv_f; oq.ldy = 3 * d;
    oh.planes = v.hp; oh.ldp = F;
    for (int l = 0; l < c.n_layer; ++l) {
        const LayerDev& L = m->layers[l];
        FC_TRY(normed(L.ln1g, L.ln1b));
        FC_TRY(launch_skinny_q8(b.qkv[l], S, v.xp, L.qkv_b, EPI_NONE, oq, nullptr, st));
        FC_TRY(launch_attn_decode_batch(v.qkv_f, v.kcs, v.vcs, l * layer_stride, d, c.n_head, c.ctx, v.pos, S, v.ap, st));
        FC_TRY(project_add(b.out[l], v.ap, L.out_b));
        FC_TRY(normed(L.ln2g, L.ln2b));
        FC_TRY(launch_skinny_q8(b.up[l], S, v.xp, L.up_b, EPI_GELU, oh, nullptr, st));
        FC_TRY(project_add(b.down[l], v.hp, L.down_b));
    }
    return batch_head_and_pick(m, v, eos, x, v.part, n_part, part_bias, x_other, 1);
}

// Streams per group of the step graph. Every step kernel is a chain of memory round trips that leaves most of the
// GPU idle, and its duration hardly falls with fewer streams, so groups run as parallel branches of the graph and
// their chains overlap. The weights are then read once per group, the re-reads coming from L2 (a block's matrices
// are a few MB and the branches stay within a block or two of each other). Measured on the 24-block, 1024-wide
// shape with 64 streams: one group 1.63 ms per step, groups of 32 1.47 ms, of 16 1.37 ms, of 8 1.55 ms.
// FERRUM_LOCKSTEP_GROUP=<n> overrides the choice (a tuning aid; results do not depend on it beyond the
// summation order of the kernels that n selects).
static int batch_group_size(int S) {
    if (const char* e = getenv("FERRUM_LOCKSTEP_GROUP")) {
        const int forced = atoi(e);
        if (forced > 0) return std::min(forced, kBatchMaxStreams);
    }
    return S > 16 ? 16 : S;
}

// All groups of one step on the capture: group 0 on the model's stream, the others on side streams forked from
// it and joined back.
static int batch_launch_groups(fc_model* m, int S, int eos, int group) {
    BatchCtx& b = m->batch;
    const int n_groups = (S + group - 1) / group;
    while ((int)b.side.size() < n_groups - 1) {
        cudaStream_t s = nullptr;
        cudaEvent_t e = nullptr;
        FC_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        b.side.push_back(s);
        FC_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        b.side_done.push_back(e);
    }
    if (!b.fork) FC_CUDA(cudaEventCreateWithFlags(&b.fork, cudaEventDisableTiming));
    if (n_groups > 1) FC_CUDA(cudaEventRecord(b.fork, m->st));
    for (int g = 1; g < n_groups; ++g) {
        FC_CUDA(cudaStreamWaitEvent(b.side[g - 1], b.fork, 0));
        FC_TRY(batch_launch_step(m, batch_view(m, g * group, std::min(group, S - g * group), g, b.side[g - 1], n_groups), eos));
        FC_CUDA(cudaEventRecord(b.side_done[g - 1], b.side[g - 1]));
    }
    FC_TRY(batch_launch_step(m, batch_view(m, 0, std::min(group, S), 0, m->st, n_groups), eos));
    for (int g = 1; g < n_groups; ++g) FC_CUDA(cudaStreamWaitEvent(m->st, b.side_done[g - 1], 0));
    return FC_OK;
}

// The step is launch-bound (7 small kernels per block): it is captured once into a CUDA graph and
// replayed; position and tokens are read from device memory, so no node changes between steps.
// n_steps: 1 or 4 consecutive steps in one launch.
static int batch_run_steps(fc_model* m, int S, int eos, int n_steps) {
    BatchCtx& b = m->batch;
    const int group = batch_group_size(S);
    if (b.graph_S != S || b.graph_eos != eos || b.graph_cap != b.out_cap || b.graph_group != group) {
        if (b.graph) { cudaGraphExecDestroy(b.graph); b.graph = nullptr; }
        if (b.graph4) { cudaGraphExecDestroy(b.graph4); b.graph4 = nullptr; }
        b.graph_S = S; b.graph_eos = eos; b.graph_cap = b.out_cap; b.graph_group = group;
    }
    cudaGraphExec_t& exec = n_steps == 4 ? b.graph4 : b.graph;
    int& nodes = n_steps == 4 ? b.graph4_nodes : b.graph_nodes;
    if (!exec) {
        cudaGraph_t g = nullptr;
        const int64_t before = g_launches;
        FC_CUDA(cudaStreamBeginCapture(m->st, cudaStreamCaptureModeThreadLocal));
        int rc = FC_OK;
        for (int k = 0; k < n_steps && rc == FC_OK; ++k) rc = batch_launch_groups(m, S, eos, group);
        const cudaError_t e = cudaStreamEndCapture(m->st, &g);
        nodes = (int)(g_launches - before);
        g_launches = before;
        if (rc != FC_OK) { if (g) cudaGraphDestroy(g); return rc; }
        FC_CUDA(e);
        const cudaError_t ei = cudaGraphInstantiate(&exec, g, 0);
        cudaGraphDestroy(g);
        FC_CUDA(ei);
    }
    FC_CUDA(cudaGraphLaunch(exec, m->st));
    g_launches += nodes;
    return FC_OK;
}

// Independent greedy streams on one GPU (the 64-stream workload is split over GPUs above the
// ABI). Each stream is a CachedTransformer of its own (its own KV caches and window); the
// streams advance in lock step, up to 64 at a time: the prompts are primed as one batch of
// windows, then every step runs all streams through each Q8_0 matrix at once, so the weights
// are read once per step whatever the number of streams. A stream that picks `eos` stops
// emitting; the others go on. The reference's extra feed after the last sampled token
// (token_stream.rs:181-186) is not run: its distribution is never used.
// Streams that would outgrow the context (they need the re-prime of token_stream.rs:162-165)
// and single streams run one after the other through fc_generate_greedy.
int fc_decode_batch(fc_model* m, int n_streams, const int32_t* prompts, int prompt_len, int max_new, int32_t eos,
                    int32_t* out, int* n_out) {
    if (!m || !prompts || !n_out || (max_new > 0 && !out)) return fail(FC_E_ARG, "fc_decode_batch: null argument");
    if (n_streams < 0 || prompt_len <= 0 || max_new < 0) return fail(FC_E_SHAPE, "fc_decode_batch: bad sizes");
    FC_CUDA(cudaSetDevice(m->device));
    const fc_config& c = m->cfg;
    while ((int)m->pool.size() < n_streams) {
        fc_stream* s = nullptr;
        FC_TRY(fc_stream_create(m, &s));
        m->pool.push_back(s);
    }
    m->last_batch_ms = 0.0f;
    m->last_batch_prime_ms = 0.0f;
    if (!m->ev_prime) FC_CUDA(cudaEventCreate(&m->ev_prime));
    const int hd = c.d_model / c.n_head;
    const bool lock_step = n_streams >= 2 && max_new > 0 && prompt_len + max_new <= c.ctx && hd <= 64 && hd % 4 == 0 &&
                           (size_t)(c.ctx + 4 + 64 + 1024) * sizeof(float) <= 48 * 1024;
    if (!lock_step) {
        for (int i = 0; i < n_streams; ++i) {
            FC_TRY(fc_generate_greedy(m->pool[i], prompts + (size_t)i * prompt_len, prompt_len, max_new, eos, nullptr,
                                      out + (size_t)i * max_new, n_out + i));
            m->last_batch_ms += m->pool[i]->last_decode_ms;
        }
        return FC_OK;
    }
    FC_TRY(check_ids(m, prompts, (size_t)n_streams * prompt_len));
    FC_TRY(with_room(m, [&] { return batch_make_frags(m); }));
    FC_TRY(with_room(m, [&] { return batch_ensure(m, std::min(n_streams, kBatchMaxStreams), max_new); }));
    BatchCtx& b = m->batch;
    cudaStream_t st = m->st;
    FC_CUDA(cudaEventRecord(m->ev0, st));
    for (int w0 = 0; w0 < n_streams; w0 += kBatchMaxStreams) {
        const int S = std::min(kBatchMaxStreams, n_streams - w0);
        if (w0 > 0) FC_CUDA(cudaEventRecord(m->ev1, st));   // start of this wave's prime (the first wave starts at ev0)
        // prime: all prompts of the wave as one batch of windows; the last row of each selects token 1
        std::vector<fc_stream*> wv;
        for (int i = 0; i < S; ++i) {
            fc_stream* s = m->pool[w0 + i];
            s->table = 0;
            FC_TRY(fc_stream_reset(s));
            FC_CUDA(cudaMemcpyAsync(s->queue, prompts + (size_t)(w0 + i) * prompt_len, (size_t)prompt_len * 4, cudaMemcpyHostToDevice, st));
            FC_TRY(set_state(s, 0, 0, prompt_len, eos, 0));
            wv.push_back(s);
        }
        // per-stream pointers for the step kernels
        std::vector<float*> kcs(S), vcs(S);
        std::vector<int*> queues(S);
        std::vector<StepState*> states(S);
        for (int i = 0; i < S; ++i) { kcs[i] = wv[i]->kc; vcs[i] = wv[i]->vc; queues[i] = wv[i]->queue; states[i] = wv[i]->state; }
        FC_CUDA(cudaMemcpyAsync(b.kcs, kcs.data(), S * sizeof(float*), cudaMemcpyHostToDevice, st));
        FC_CUDA(cudaMemcpyAsync(b.vcs, vcs.data(), S * sizeof(float*), cudaMemcpyHostToDevice, st));
        FC_CUDA(cudaMemcpyAsync(b.queues, queues.data(), S * sizeof(int*), cudaMemcpyHostToDevice, st));
        FC_CUDA(cudaMemcpyAsync(b.states, states.data(), S * sizeof(StepState*), cudaMemcpyHostToDevice, st));
        FC_CUDA(cudaStreamSynchronize(st));   // the host vectors above go out of use
        int used = 0;
        FC_TRY(prime_batched(wv.data(), S, prompt_len, STEP_NOHEAD, &used, b.kcs, b.vcs));
        if (used) {
            // the head sees the last row of every window: final LayerNorm, one product for all streams, pick of token 1
            const int d = c.d_model;
            FC_TRY(launch_gather_last_rows(m->x, S, prompt_len, d, b.x, st));
            FC_TRY(launch_batch_init(S, prompt_len, m->tc_status, b.done, b.n_out, b.cur, b.pos, st));
            FC_TRY(batch_head_and_pick(m, batch_view(m, 0, S, 0, st), eos, b.x, nullptr, 0, nullptr, nullptr, 0));
        } else {
            // prompts too short for a window forward: token by token per stream; the last step selects token 1
            for (int i = 0; i < S; ++i) {
                StepState hs;
                FC_TRY(run_steps(wv[i], prompt_len, STEP_NOHEAD, STEP_SELECT, 0));
                FC_TRY(read_state(wv[i], &hs));
            }
            FC_TRY(launch_gather_first(b.queues, b.states, prompt_len, S, b.cur, b.done, b.n_out, b.out_tok, b.out_cap, b.pos, st));
        }
        FC_CUDA(cudaEventRecord(m->ev_prime, st));
        std::vector<int> done(S, 0);
        for (int i = 1; i < max_new; ++i) {        // step i feeds token i and picks token i + 1
            // four steps per launch while they fit (steps 1-4, 5-8, ...: a chunk ends where the eos check falls)
            const int n_steps = (i % 4 == 1 && i + 3 < max_new) ? 4 : 1;
            FC_TRY(batch_run_steps(m, S, eos, n_steps));
            i += n_steps - 1;
            if (eos >= 0 && (i % 16 == 0)) {          // eos can only be noticed on the host at a synchronisation point
                FC_CUDA(cudaMemcpyAsync(done.data(), b.done, S * sizeof(int), cudaMemcpyDeviceToHost, st));
                FC_CUDA(cudaStreamSynchronize(st));
                if (std::all_of(done.begin(), done.end(), [](int v) { return v != 0; })) break;
            }
        }
        std::vector<int> cnt(S);
        FC_CUDA(cudaMemcpyAsync(done.data(), b.done, S * sizeof(int), cudaMemcpyDeviceToHost, st));
        std::vector<int32_t> toks((size_t)S * b.out_cap);
        int pos_h = 0;
        FC_CUDA(cudaMemcpyAsync(cnt.data(), b.n_out, S * sizeof(int), cudaMemcpyDeviceToHost, st));
        FC_CUDA(cudaMemcpyAsync(toks.data(), b.out_tok, toks.size() * 4, cudaMemcpyDeviceToHost, st));
        FC_CUDA(cudaMemcpyAsync(&pos_h, b.pos, sizeof(int), cudaMemcpyDeviceToHost, st));
        FC_CUDA(cudaStreamSynchronize(st));
        {
            float pm = 0.0f;
            FC_CUDA(cudaEventElapsedTime(&pm, w0 > 0 ? m->ev1 : m->ev0, m->ev_prime));
            m->last_batch_prime_ms += pm;
        }
        if (done[0] == 3) return check_tc_status(m, "the prime of fc_decode_batch");
        for (int i = 0; i < S; ++i)
            if (done[i] == 2) return fail(FC_E_CUDA, "fc_decode_batch: stream %d produced no finite logit", w0 + i);
        for (int i = 0; i < S; ++i) {
            const int have = std::min(cnt[i], max_new);
            std::copy(toks.begin() + (size_t)i * b.out_cap, toks.begin() + (size_t)i * b.out_cap + have, out + (size_t)(w0 + i) * max_new);
            n_out[w0 + i] = have;
            wv[i]->host_pos = pos_h;
        }
    }
    FC_CUDA(cudaEventRecord(m->ev1, st));
    FC_CUDA(cudaStreamSynchronize(st));
    FC_CUDA(cudaEventElapsedTime(&m->last_batch_ms, m->ev0, m->ev1));
    return FC_OK;
}

float fc_last_batch_ms(const fc_model* m) { return m ? m->last_batch_ms : 0.0f; }
float fc_last_batch_prime_ms(const fc_model* m) { return m ? m->last_batch_prime_ms : 0.0f; }

}  // extern "C"

// ---------------------------------------------------------------- several devices, one call
namespace {
// Runs fn(i, first, last) for every model on a host thread of its own (one handle = one GPU = one host thread
// at a time, as everywhere in this ABI), item i * n / n_models .. (i + 1) * n / n_models each. The first
// failure (in model order) is returned with its message; kernel launches are credited to the caller.
template <class Fn>
int run_on_models(int n_models, int n_items, Fn fn) {
    std::vector<int> rc(n_models, FC_OK);
    std::vector<std::string> msg(n_models);
    std::vector<int64_t> launches(n_models, 0);
    std::vector<std::thread> workers;
    for (int i = 0; i < n_models; ++i) {
        const int first = (int)((long long)i * n_items / n_models), last = (int)((long long)(i + 1) * n_items / n_models);
        workers.emplace_back([&, i, first, last] {
            if (last > first) rc[i] = fn(i, first, last);
            if (rc[i] != FC_OK) msg[i] = fc::g_err_text();
            launches[i] = fc::g_launches;
        });
    }
    for (auto& w : workers) w.join();
    for (int i = 0; i < n_models; ++i) fc::g_launches += launches[i];
    for (int i = 0; i < n_models; ++i)
        if (rc[i] != FC_OK) return fail(rc[i], "model %d of %d: %s", i, n_models, msg[i].c_str());
    return FC_OK;
}
}  // namespace

extern "C" {

int fc_score_sequences_multi(fc_model* const* models, int n_models, const int32_t* ids, int n_seq, int seq_len, int batch_windows,
                             fc_score* scores, float* lp) {
    if (!models || n_models <= 0 || !ids || !scores) return fail(FC_E_ARG, "fc_score_sequences_multi: null argument");
    for (int i = 0; i < n_models; ++i)
        if (!models[i]) return fail(FC_E_ARG, "fc_score_sequences_multi: model %d is null", i);
    if (n_seq < 0 || seq_len < 0) return fail(FC_E_SHAPE, "fc_score_sequences_multi: negative size");
    return run_on_models(n_models, n_seq, [&](int i, int a, int b) {
        return fc_score_sequences(models[i], ids + (size_t)a * seq_len, b - a, seq_len, batch_windows, scores + a,
                                  lp ? lp + (size_t)a * seq_len : nullptr);
    });
}

int fc_decode_batch_multi(fc_model* const* models, int n_models, int n_streams, const int32_t* prompts, int prompt_len, int max_new,
                          int32_t eos, int32_t* out, int* n_out) {
    if (!models || n_models <= 0 || !prompts || !n_out || (max_new > 0 && !out)) return fail(FC_E_ARG, "fc_decode_batch_multi: null argument");
    for (int i = 0; i < n_models; ++i)
        if (!models[i]) return fail(FC_E_ARG, "fc_decode_batch_multi: model %d is null", i);
    if (n_streams < 0 || prompt_len <= 0 || max_new < 0) return fail(FC_E_SHAPE, "fc_decode_batch_multi: bad sizes");
    return run_on_models(n_models, n_streams, [&](int i, int a, int b) {
        return fc_decode_batch(models[i], b - a, prompts + (size_t)a * prompt_len, prompt_len, max_new, eos, out + (size_t)a * max_new, n_out + a);
    });
}

int fc_debug_withhold_scratch(int on) {
    g_debug.withhold_scratch = on == 2 ? 2 : on != 0;
    return FC_OK;
}

int fc_debug_set_wait_budget(long long cycles, int withhold_producers) {
    if (cycles <= 0) return fail(FC_E_ARG, "fc_debug_set_wait_budget: cycles = %lld", cycles);
    g_debug.wait_cycles = cycles;
    g_debug.withhold = withhold_producers == 2 ? 2 : withhold_producers != 0;
    return FC_OK;
}

}  // extern "C"
