// Row kernels of the forward path: embedding gather, LayerNorm, the decode tail
// (probabilities or greedy select behind a head that left statistics) and the layer statistics.

#include <algorithm>

#include "pdl.cuh"
#include "planes.cuh"

namespace fc {

// ------------------------------------------------------------------------ block reductions
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
// Fixed-order block reductions (deterministic run to run). `red` has >= 33 floats.
__device__ float block_sum(float v, float* red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (wid == 0) {
        float t = lane < nw ? red[lane] : 0.0f;
        t = warp_sum(t);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}
__device__ float block_max(float v, float* red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (wid == 0) {
        float t = lane < nw ? red[lane] : -INFINITY;
        t = warp_max(t);
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

// ------------------------------------------------------------------------------ embedding
// layer/embedding.rs:70-90 embed_one / :98-152 forward: x = tok[id] + pos[t]. The token
// table stays Q8_0; d * q is the same single rounding gguf::dequant_q8_0 performs.
__device__ __forceinline__ float tok_value(const QMat& tok, int id, int c) {
    const float dq = __half2float(tok.d[(size_t)id * (tok.K >> 5) + (c >> 5)]);
    const int q = (int)tok.qu[(size_t)id * tok.K + c] - 128;
    return dq * (float)q;
}

__global__ void embed_step_kernel(QMat tok, const float* __restrict__ pos_emb, int ctx,
                                  const int* __restrict__ queue, StepState* st, float* __restrict__ x) {
    pdl_wait();
    pdl_trigger();       // only now: the chain's attention reads state and caches ahead of its own wait
    if (st->done | st->error) return;
    const int pos = st->pos, id = queue[st->fed];
    // embedding.rs:71-82 and transformer.rs:237-242: bad id / full cache are errors, not traps
    if (id < 0 || id >= tok.N || pos >= ctx) {
        __syncthreads();
        if (threadIdx.x == 0) st->error = FC_E_DIM;
        return;
    }
    for (int c = threadIdx.x; c < tok.K; c += blockDim.x) x[c] = tok_value(tok, id, c) + pos_emb[(size_t)pos * tok.K + c];
}

int launch_embed_step(const QMat& tok, const float* pos_emb, int ctx, const int* queue, StepState* state,
                      float* x, cudaStream_t st) {
    FC_CUDA(launch_pdl(embed_step_kernel, dim3(1), dim3(256), 0, st, tok, pos_emb, ctx, queue, state, x));
    ++g_launches;
    return FC_OK;
}

__global__ void embed_rows_kernel(QMat tok, const float* __restrict__ pos_emb, const int* __restrict__ ids, const int* __restrict__ pos,
                                  int T, float* __restrict__ x, int* error_flag) {
    const int r = blockIdx.x, t = pos ? pos[r] : r % T;
    int id = ids[r];
    if (id < 0 || id >= tok.N) {
        if (threadIdx.x == 0) atomicExch(error_flag, FC_E_DIM);
        id = 0;
    }
    for (int c = threadIdx.x; c < tok.K; c += blockDim.x)
        x[(size_t)r * tok.K + c] = tok_value(tok, id, c) + pos_emb[(size_t)t * tok.K + c];
}

int launch_embed_rows(const QMat& tok, const float* pos_emb, const int* ids, const int* pos, int R, int T, float* x,
                      int* error_flag, cudaStream_t st) {
    embed_rows_kernel<<<R, 256, 0, st>>>(tok, pos_emb, ids, pos, T, x, error_flag);
    FC_LAUNCHED();
    return FC_OK;
}

// ------------------------------------------------------------------------------ LayerNorm
// layer/norm.rs:46-82: mean, then the variance of (x - mean), std = sqrt(var + 1e-5),
// y = ((x - mean) / std) * gamma + beta. One block per row; the row is held in registers.
// The result is written as the P bf16 planes that the tensor-core GEMM reads.
template <int PER, int P>
__global__ void layernorm_planes_kernel(const float* __restrict__ x, const float* __restrict__ g, const float* __restrict__ b,
                                        const int* __restrict__ pick, int d, const Planes out) {
    __shared__ float red[33];
    pdl_wait();
    pdl_trigger();
    const float* xr = x + (size_t)(pick ? pick[blockIdx.x] : (int)blockIdx.x) * d;
    float v[PER];
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        v[i] = c < d ? xr[c] : 0.0f;
        s += v[i];
    }
    const float mean = block_sum(s, red) / (float)d;
    float q = 0.0f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        const float t = v[i] - mean;
        q += c < d ? t * t : 0.0f;
    }
    const float var = block_sum(q, red) / (float)d;
    const float sd = sqrtf(var + 1e-5f);
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int c = threadIdx.x + i * blockDim.x;
        if (c < d) store_planes<P>(out, (size_t)blockIdx.x * d + c, ((v[i] - mean) / sd) * g[c] + b[c]);
    }
}

// The same for rows of up to 1024 columns (a multiple of 128): a warp per row, the row in registers as 16-byte loads,
// the two sums by shuffles (no block-wide synchronisation), the planes written 8 bytes per lane. Eight rows per CTA.
template <int NV, int P>
__global__ void __launch_bounds__(256) layernorm_planes_warp_kernel(const float* __restrict__ x, const float* __restrict__ g,
                                                                    const float* __restrict__ b, const int* __restrict__ pick, int rows,
                                                                    int d, const Planes out) {
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    pdl_wait();
    pdl_trigger();
    if (row >= rows) return;
    const int nv = d >> 7;                                  // 16-byte chunks per lane
    const float4* xr = (const float4*)(x + (size_t)(pick ? pick[row] : row) * d);
    float4 v[NV];
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        v[i] = i < nv ? xr[lane + 32 * i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    const float mean = s / (float)d;
    float q = 0.0f;
#pragma unroll
    for (int i = 0; i < NV; ++i)
        if (i < nv) {
            const float a = v[i].x - mean, c = v[i].y - mean, e = v[i].z - mean, f = v[i].w - mean;
            q += (a * a + c * c) + (e * e + f * f);
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
    const float sd = sqrtf(q / (float)d + 1e-5f);
    const float4* g4 = (const float4*)g;
    const float4* b4 = (const float4*)b;
#pragma unroll
    for (int i = 0; i < NV; ++i)
        if (i < nv) {
            const float4 gg = __ldg(g4 + lane + 32 * i), bb = __ldg(b4 + lane + 32 * i);
            store_planes4<P>(out, (size_t)row * (d >> 2) + lane + 32 * i,
                             make_float4(((v[i].x - mean) / sd) * gg.x + bb.x, ((v[i].y - mean) / sd) * gg.y + bb.y,
                                         ((v[i].z - mean) / sd) * gg.z + bb.z, ((v[i].w - mean) / sd) * gg.w + bb.w));
        }
}

template <int P>
static int layernorm_planes(const float* x, const float* g, const float* b, const int* pick, int rows, int d, const Planes& out,
                            cudaStream_t st) {
    if (d % 128 == 0 && d <= 1024 && aligned16(x) && aligned16(g) && aligned16(b)) {
        const int blocks = (rows + 7) / 8;
        FC_CUDA(launch_pdl(d <= 512 ? layernorm_planes_warp_kernel<4, P> : layernorm_planes_warp_kernel<8, P>, dim3(blocks), dim3(256), 0, st, x, g, b, pick, rows, d, out));
        FC_LAUNCHED();
        return FC_OK;
    }
    const int threads = 256;
    const int per = (d + threads - 1) / threads;
    if (per > 16) return fail(FC_E_SHAPE, "LayerNorm width %d exceeds 4096", d);
    FC_CUDA(launch_pdl(per <= 4 ? layernorm_planes_kernel<4, P> : per <= 8 ? layernorm_planes_kernel<8, P> : layernorm_planes_kernel<16, P>, dim3(rows),
                       dim3(threads), 0, st, x, g, b, pick, d, out));
    FC_LAUNCHED();
    return FC_OK;
}
int launch_layernorm_planes(const float* x, const float* g, const float* b, const int* pick, int rows, int d, const Planes& out,
                            cudaStream_t st) {
    if (out.scale != 0.0f) return layernorm_planes<F16X2>(x, g, b, pick, rows, d, out, st);
    return out.n == 3 ? layernorm_planes<3>(x, g, b, pick, rows, d, out, st) : layernorm_planes<2>(x, g, b, pick, rows, d, out, st);
}

// ------------------------------------------------------------------------------ decode tail
// ops.rs:478-502 softmax_rows on one row, then (when selecting) token_stream.rs:134 +
// sampling.rs:96-104,147: logit_i = ln(max(p_i, 1e-12)), first index of the largest.
// One block. The sum runs in a fixed tree order, not the reference's ascending order.
struct ArgPair { float v; int i; };
__device__ __forceinline__ ArgPair better(ArgPair a, ArgPair b) {
    // larger value wins; equal values: smaller index (first on ties)
    return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}

// The tail of a step whose head product left, per CTA, its largest logit and the mass around it: the softmax needs no pass of
// its own. M and S of the whole row, by every warp for itself.
__device__ __forceinline__ float2 row_stats(const float2* __restrict__ stats, int n) {
    const int lane = threadIdx.x & 31;
    float top = -INFINITY, mass = 0.0f;
    for (int i = lane; i < n; i += 32) {
        const float2 s = stats[i];
        if (s.x > top) { mass *= expf(top - s.x); top = s.x; }
        if (s.y != 0.0f) mass += s.y * expf(s.x - top);
    }
    float all = top;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) all = fmaxf(all, __shfl_xor_sync(0xffffffffu, all, o));
    mass = mass != 0.0f ? mass * expf(top - all) : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, o);
    return make_float2(all, mass);
}
// Greedy pick: first index of the largest ln(max(p, 1e-12)). Rounding can make neighbours of the largest logit tie with it, but
// nothing 0.01 below it (p there is at least 1 % smaller, and the largest p is at least 1 / V), so only those are evaluated.
// A row with a NaN or an infinity, or of -inf alone, has no mass to compare: every p is NaN, all tie at the floor, the first wins.
// span: stats[c] is over the rows of which (row / span) % n_stats is c (launch_head_row), so only where a largest one reaches the bound are logits
// read: some 340 of 50257, behind the statistics, in place of a pass of one SM over the row
// (a token of 12 x 768 129.7 us, now 129.0). 0: stats says nothing of rows.
__global__ void __launch_bounds__(1024) step_pick_kernel(const float* __restrict__ logits, int V, const float2* __restrict__ stats, int n_stats, int span,
                                                         int* __restrict__ queue, int queue_cap, StepState* st) {
    __shared__ ArgPair pred[32];
    pdl_trigger();
    pdl_wait();
    if (st->done | st->error) return;
    const float2 ms = row_stats(stats, n_stats);
    ArgPair best{-INFINITY, 0x7fffffff};
    auto look = [&](float l, int i) {
        if (l >= ms.x - 0.01f) best = better(best, ArgPair{logf(fmaxf(expf(l - ms.x) / ms.y, 1e-12f)), i});
    };
    const bool comparable = ms.y > 0.0f;
    if (!comparable) best = ArgPair{0.0f, 0};
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int c = wid; span && comparable && c < n_stats; c += 32) {
        if (stats[c].x < ms.x - 0.01f) continue;
        const int stride = n_stats * span;
        for (int i0 = c * span; i0 < V; i0 += 12 * stride) {
            for (int j = lane; j < span; j += 32) {
                float l[12];             // on their way at a time: all of 50257 over 148
#pragma unroll
                for (int k = 0; k < 12; ++k) l[k] = i0 + k * stride + j < V ? logits[i0 + k * stride + j] : -INFINITY;
#pragma unroll
                for (int k = 0; k < 12; ++k) look(l[k], i0 + k * stride + j);
            }
        }
    }
    const bool whole = comparable && !span;
    const int V4 = whole ? V >> 2 : 0;
    for (int i0 = threadIdx.x; i0 < V4; i0 += 7 * blockDim.x) {
        float4 l[7];                     // 28 K logits on their way at a time
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const int i = i0 + k * blockDim.x;
            l[k] = i < V4 ? ((const float4*)logits)[i] : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        }
#pragma unroll
        for (int k = 0; k < 7; ++k) {
            const int i = 4 * (i0 + k * blockDim.x);
            if (fmaxf(fmaxf(l[k].x, l[k].y), fmaxf(l[k].z, l[k].w)) < ms.x - 0.01f) continue;
            look(l[k].x, i); look(l[k].y, i + 1); look(l[k].z, i + 2); look(l[k].w, i + 3);
        }
    }
    if (whole && (int)threadIdx.x < (V & 3)) look(logits[4 * V4 + threadIdx.x], 4 * V4 + threadIdx.x);
    auto warp_best = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            best = better(best, ArgPair{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
    };
    warp_best();
    if (lane == 0) pred[wid] = best;
    __syncthreads();
    if (wid != 0) return;
    best = pred[lane];
    warp_best();
    if (lane != 0) return;
    if (best.i == st->eos) {
        st->done = 1;
    } else if (st->tail < queue_cap) {
        queue[st->tail] = best.i;
        st->tail += 1;
    } else {
        st->error = FC_E_DIM;
    }
    st->pos += 1;
    st->fed += 1;
}
__global__ void __launch_bounds__(256) step_probs_kernel(const float* __restrict__ logits, int V, const float2* __restrict__ stats, int n_stats,
                                                         float* __restrict__ probs, StepState* st) {
    pdl_trigger();
    pdl_wait();
    if (st->done | st->error) return;
    const float2 ms = row_stats(stats, n_stats);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < V; i += gridDim.x * blockDim.x) probs[i] = expf(logits[i] - ms.x) / ms.y;
    if (blockIdx.x == 0 && threadIdx.x == 0) { st->pos += 1; st->fed += 1; }
}
int launch_step_finish(const float* logits, int V, const float2* stats, int n_stats, int span, float* probs_or_null, int* queue, int queue_cap,
                       StepState* state, cudaStream_t st) {
    if (probs_or_null)
        FC_CUDA(launch_pdl(step_probs_kernel, dim3(std::min(148, (V + 255) / 256)), dim3(256), 0, st, logits, V, stats, n_stats, probs_or_null, state));
    else
        FC_CUDA(launch_pdl(step_pick_kernel, dim3(1), dim3(1024), 0, st, logits, V, stats, n_stats, span, queue, queue_cap, state));
    ++g_launches;
    return FC_OK;
}

__global__ void step_advance_kernel(StepState* st) {
    pdl_trigger();
    pdl_wait();
    if (st->done | st->error) return;
    st->pos += 1;
    st->fed += 1;
}
// A programmatic dependent of the kernel ahead (steps whose kernels all wait first).
int launch_step_advance_pdl(StepState* state, cudaStream_t st) {
    FC_CUDA(launch_pdl(step_advance_kernel, dim3(1), dim3(1), 0, st, state));
    ++g_launches;
    return FC_OK;
}

__global__ void __launch_bounds__(1024) softmax_row_kernel(const float* __restrict__ logits, int V, float* __restrict__ probs) {
    __shared__ float red[33];
    float mx = -INFINITY;
    for (int i = threadIdx.x; i < V; i += blockDim.x) mx = fmaxf(mx, logits[i]);
    mx = block_max(mx, red);
    float s = 0.0f;
    for (int i = threadIdx.x; i < V; i += blockDim.x) s += expf(logits[i] - mx);
    const float sum = block_sum(s, red);
    for (int i = threadIdx.x; i < V; i += blockDim.x) probs[i] = expf(logits[i] - mx) / sum;
}
int launch_softmax_row(const float* logits, int V, float* probs, cudaStream_t st) {
    softmax_row_kernel<<<1, 1024, 0, st>>>(logits, V, probs);
    FC_LAUNCHED();
    return FC_OK;
}

// ------------------------------------------------------------------------------ layer statistics
// verbose::stats + verbose::check_nan_inf (verbose.rs:85-110) of one layer output: min, max, f64 sum, and the
// counts of NaN and Inf. Two stages with a fixed order (per-block partials, then one block), so the figures are
// the same from run to run. x == null: the tensor is held as bf16 planes, value = their sum.
struct StatPart { float mn, mx; double sum; unsigned long long nan, inf; };

__global__ void __launch_bounds__(256) layer_stats_partial_kernel(const float* __restrict__ x, const Planes pl, size_t n, StatPart* part) {
    __shared__ StatPart sh[256];
    StatPart p{INFINITY, -INFINITY, 0.0, 0ull, 0ull};
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        float v = 0.0f;
        if (x) v = x[i];
        else
            for (int p = pl.n - 1; p >= 0; --p) v += __bfloat162float(((const __nv_bfloat16*)pl.p[p])[i]);
        if (v != v) { p.nan += 1; continue; }      // as the reference's comparisons, NaN never becomes min or max
        if (isinf(v)) p.inf += 1;
        p.mn = fminf(p.mn, v);
        p.mx = fmaxf(p.mx, v);
        p.sum += (double)v;
    }
    sh[threadIdx.x] = p;
    __syncthreads();
    if (threadIdx.x == 0) {
        StatPart t = sh[0];
        for (int i = 1; i < (int)blockDim.x; ++i) {
            t.mn = fminf(t.mn, sh[i].mn); t.mx = fmaxf(t.mx, sh[i].mx); t.sum += sh[i].sum; t.nan += sh[i].nan; t.inf += sh[i].inf;
        }
        part[blockIdx.x] = t;
    }
}

__global__ void layer_stats_final_kernel(const StatPart* part, int n_part, size_t n, LayerStatsDev* out) {
    StatPart t = part[0];
    for (int i = 1; i < n_part; ++i) {
        t.mn = fminf(t.mn, part[i].mn); t.mx = fmaxf(t.mx, part[i].mx); t.sum += part[i].sum; t.nan += part[i].nan; t.inf += part[i].inf;
    }
    out->min = n ? t.mn : 0.0f;
    out->max = n ? t.mx : 0.0f;
    out->mean = n ? (float)(t.sum / (double)n) : 0.0f;
    out->nan_count = (long long)t.nan;
    out->inf_count = (long long)t.inf;
    out->n = (long long)n;
}

size_t layer_stats_scratch_bytes() { return 148 * sizeof(StatPart); }

int launch_layer_stats(const float* x, const Planes& planes, size_t n, void* scratch, LayerStatsDev* out, cudaStream_t st) {
    const int blocks = (int)std::min<size_t>(148, std::max<size_t>(1, (n + 255) / 256));
    layer_stats_partial_kernel<<<blocks, 256, 0, st>>>(x, planes, n, (StatPart*)scratch);
    FC_LAUNCHED();
    layer_stats_final_kernel<<<1, 1, 0, st>>>((const StatPart*)scratch, blocks, n, out);
    FC_LAUNCHED();
    return FC_OK;
}

}  // namespace fc
