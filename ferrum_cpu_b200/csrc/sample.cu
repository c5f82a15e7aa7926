// Token sampler on the device: repetition penalty -> temperature softmax -> top-k -> top-p ->
// renormalise -> inverse-CDF draw, the pipeline of sample_with_params
// (ferrum_core/src/slm/sampling.rs:124-210) on the log-probabilities stream_next builds
// (slm/token_stream.rs:134: ln(max(p, 1e-12))), with Ferrum's xorshift64* generator
// (rng.rs:29-40) advanced on the device.
//
// One CTA, the row staged in shared memory, or eight that share the passes over a long row. Differences from the sequential reference, all at
// rounding level: sums are block reductions (a different association than index order), the
// running mass of the draw is a block scan + a sequential walk inside one thread's chunk, and
// probabilities that tie exactly at the top-p cut are all kept (the reference's unstable sort
// keeps an unspecified subset of them). A draw can therefore differ from the reference only
// when r falls within rounding of a cumulative boundary.
//
// Bound: latency of one CTA: a row of V floats in shared memory costs V / 32 cycles a pass (0.8 us at V = 50257). Finding the
// cuts by bisection of their bit patterns takes 31 such passes each (155 us a draw at V = 50257 with top-k 40 and top-p 0.95).
// With a top-k of at most kListK the row is therefore passed five times only: the k-th largest of the threads' maxima bounds
// the k-th largest value from below, and the few values that reach it go to a list on which every later step works: a
// draw at V = 50257 with top-k 40 takes 24.9 us.
#include <cooperative_groups.h>

#include <climits>

#include "fc_common.cuh"

namespace fc {

namespace {
constexpr int ST = 1024;       // threads
constexpr int kList = 1024;    // candidates the list holds
// Up to half as many as there are thread maxima: above that the bound drops into the bulk of a flat row and the list overflows.
constexpr int kListK = 512;
constexpr int kSampleMax = 51200;   // values of a row that shared memory holds
constexpr int kClusterRow = 8192;   // values from which they do
constexpr int kCluster = 8;         // CTAs that share the passes over a row

__device__ float bsum(float v, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < ST / 32; ++w) t += red[w];
    return t;
}
__device__ float bmax(float v, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = -INFINITY;
#pragma unroll
    for (int w = 0; w < ST / 32; ++w) t = fmaxf(t, red[w]);
    return t;
}
__device__ int bsum_int(int v, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = __int_as_float(v);
    __syncthreads();
    int t = 0;
#pragma unroll
    for (int w = 0; w < ST / 32; ++w) t += __float_as_int(red[w]);
    return t;
}
// rng.rs:29-35
__device__ unsigned long long next_u64(unsigned long long* state) {
    unsigned long long x = *state;
    x ^= x << 13;
    x ^= x >> 7;
    x ^= x << 17;
    *state = x;
    return x * 0x2545F4914F6CDD1DULL;
}
// The rest of the pipeline on the n candidates of a top-k draw: (value, index) pairs in v / at, unordered, that contain every
// value the top-k may keep. O(n^2 / ST) reads of shared memory, broadcast. sv / si: the list in index order.
__device__ int draw_from_list(int n, float sum, const fc_sampling& prm, float* v, int* at, float* sv, int* si, float* red,
                              unsigned long long* rng_state) {
    __shared__ float r_draw;
    __shared__ int found;
    const int tid = threadIdx.x, n4 = (n + 3) & ~3;
    if (tid == 0) {
        r_draw = (float)(next_u64(rng_state) >> 40) / 16777216.0f;   // rng.rs:37-40
        found = 0x7fffffff;
    }
    for (int q = n + tid; q < n4; q += ST) { v[q] = -1.0f; at[q] = 0x7fffffff; sv[q] = 0.0f; si[q] = 0x7fffffff; }
    __syncthreads();
    // 3. top-k: a value stays when fewer than k are larger, by quotient, as the filter sees them
    float p = 0.0f;
    if (tid < n) v[tid] = p = v[tid] / sum;
    __syncthreads();
    if (tid < n) {
        const int mine = at[tid];
        int rank = 0, larger = 0;
        for (int q = 0; q < n4; q += 4) {
            const float4 o = *(const float4*)(v + q);
            const int4 i = *(const int4*)(at + q);
            rank += (i.x < mine) + (i.y < mine) + (i.z < mine) + (i.w < mine);
            larger += (o.x > p) + (o.y > p) + (o.z > p) + (o.w > p);
        }
        sv[rank] = larger < prm.top_k ? p : 0.0f;
        si[rank] = mine;
    }
    __syncthreads();
    p = tid < n ? sv[tid] : 0.0f;
    // 4. top-p: the largest value down to which the mass reaches top_p
    if (prm.top_p < 1.0f) {
        float mass = 0.0f;
        if (p > 0.0f)
            for (int q = 0; q < n4; q += 4) {
                const float4 o = *(const float4*)(sv + q);
                mass += ((o.x >= p ? o.x : 0.0f) + (o.y >= p ? o.y : 0.0f)) + ((o.z >= p ? o.z : 0.0f) + (o.w >= p ? o.w : 0.0f));
            }
        const float cut = bmax(p > 0.0f && mass >= prm.top_p ? p : 0.0f, red);
        if (p < cut) p = 0.0f;
        if (tid < n) sv[tid] = p;
        __syncthreads();
    }
    // 5. renormalise and draw: the mass in index order, as pick_by_mass adds it (sampling.rs:106-121)
    const float sum2 = bsum(p, red);
    p /= sum2;
    if (tid < n) sv[tid] = p;
    __syncthreads();
    if (p > 0.0f) {
        float cum = 0.0f;
        int q = 0;
#pragma unroll 4
        for (; q + 3 <= tid; q += 4) {
            const float4 o = *(const float4*)(sv + q);
            cum += o.x; cum += o.y; cum += o.z; cum += o.w;
        }
        for (; q <= tid; ++q) cum += sv[q];
        if (r_draw <= cum) atomicMin(&found, tid);
    }
    __syncthreads();
    if (found != 0x7fffffff) return si[found];
    // rounding left the total a hair under r: the last index that has any mass
    return max(0, (int)bmax(p > 0.0f ? (float)si[tid] : -1.0f, red));
}
// total order of slm/sampling.rs:96-104 (f32::total_cmp) as a signed key
__device__ __forceinline__ int order_key(float f) {
    const int b = __float_as_int(f);
    return b ^ (int)(((unsigned)(b >> 31)) >> 1);
}
}  // namespace

namespace {
struct Lists {
    __align__(16) float v[kList], sv[kList];
    __align__(16) int at[kList], si[kList];
};
__device__ __forceinline__ float logit_of(float v, int from_probs) { return from_probs ? logf(fmaxf(v, 1e-12f)) : v; }

// 1. repetition penalty, once per occurrence: the thread that holds the first occurrence of an id applies it as many times as
// the id occurs. slot(id): where its logit lies, negative for an id that is another CTA's. n_recent and rp are uniform.
template <class Slot>
__device__ void penalise(float* w, int V, float rp, const int* recent, int n_recent, int* staging, const Slot& slot) {
    if (!(fabsf(rp - 1.0f) > 1.1920929e-7f && rp > 0.0f)) return;
    const int tid = threadIdx.x;
    // a window of up to kList ids is read from shared memory, four at a time
    const bool staged = n_recent <= kList;
    const int n4 = staged ? (n_recent + 3) & ~3 : 0;
    if (staged) {
        for (int q = tid; q < n4; q += ST) staging[q] = q < n_recent ? recent[q] : -1;
        __syncthreads();
    }
    for (int j = tid; j < n_recent; j += ST) {
        const int tok = recent[j];
        if (tok < 0 || tok >= V || slot(tok) < 0) continue;
        int before = 0, count = 0;
        for (int q = 0; q < n4; q += 4) {
            const int4 o = *(const int4*)(staging + q);
            const int a = o.x == tok, b = o.y == tok, c = o.z == tok, e = o.w == tok;
            before += (a & (q < j)) + (b & (q + 1 < j)) + (c & (q + 2 < j)) + (e & (q + 3 < j));
            count += a + b + c + e;
        }
        for (int q = 0; !staged && q < n_recent; ++q) {
            const int a = recent[q] == tok;
            before += a & (q < j);
            count += a;
        }
        if (before) continue;
        float l = w[slot(tok)];
        for (int c = 0; c < count; ++c) l = l > 0.0f ? l / rp : l * rp;
        w[slot(tok)] = l;
    }
    __syncthreads();
}

// The k-th largest of the threads' maxima: at least k values reach it. A few units in the last place below it, so that whatever
// ties with it after the division by the sum is in the list too.
__device__ unsigned list_bound(float top, int k) {
    unsigned T = 0;
    for (int bit = 30; bit >= 0; --bit)
        if (__syncthreads_count(__float_as_uint(top) >= (T | (1u << bit))) >= k) T |= 1u << bit;
    return max(T, 5u) - 4;
}

// One CTA, the row in w [V].
__device__ __forceinline__ int sample_row(const float* __restrict__ in, int V, int from_probs, const fc_sampling& prm, const int* __restrict__ recent, int n_recent,
                          unsigned long long* rng_state, float* w, Lists& lists, float* red) {
    __shared__ int found;
    __shared__ float r_draw;
    __shared__ int listed;
    const int tid = threadIdx.x;
    float *lv = lists.v, *lsv = lists.sv;
    int *li = lists.at, *lsi = lists.si;

    const auto logit = [&](float v) { return logit_of(v, from_probs); };
    const int V4 = ((uintptr_t)in & 15) ? 0 : V >> 2;        // a stream's buffers are aligned, a caller's pointer may not be
#pragma unroll 4
    for (int i = tid; i < V4; i += ST) {
        const float4 v = ((const float4*)in)[i];
        ((float4*)w)[i] = make_float4(logit(v.x), logit(v.y), logit(v.z), logit(v.w));
    }
    for (int i = 4 * V4 + tid; i < V; i += ST) w[i] = logit(in[i]);
    if (tid == 0) listed = 0;
    __syncthreads();
    penalise(w, V, prm.repetition_penalty, recent, n_recent, li, [](int id) { return id; });
    int token = 0;
    if (prm.temperature <= 0.0f) {
        // argmax_first over the penalised logits; no draw
        int bk = INT_MIN, bi = 0x7fffffff;
        for (int i = tid; i < V; i += ST) {
            const int kx = order_key(w[i]);
            if (kx > bk) { bk = kx; bi = i; }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int ok = __shfl_xor_sync(0xffffffffu, bk, o), oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ok > bk || (ok == bk && oi < bi)) { bk = ok; bi = oi; }
        }
        __shared__ int kk[ST / 32], ii[ST / 32];
        if ((tid & 31) == 0) { kk[tid >> 5] = bk; ii[tid >> 5] = bi; }
        __syncthreads();
        bk = kk[0]; bi = ii[0];
        for (int q = 1; q < ST / 32; ++q)
            if (kk[q] > bk || (kk[q] == bk && ii[q] < bi)) { bk = kk[q]; bi = ii[q]; }
        token = V > 0 && bi < V ? bi : 0;
    } else {
        const float t = fmaxf(prm.temperature, 0.01f);
        // 2. temperature softmax
        float mx = -INFINITY;
        for (int i = tid; i < V; i += ST) mx = fmaxf(mx, w[i]);
        mx = bmax(mx, red);
        float s = 0.0f, top = 0.0f;
#pragma unroll 4
        for (int i = tid; i < V; i += ST) {
            const float e = expf((w[i] - mx) / t);
            w[i] = e;
            s += e;
            top = fmaxf(top, e);
        }
        const float sum = bsum(s, red);
        const bool cut_k = prm.top_k > 0 && prm.top_k < V;
        int n_list = kList + 1;
        if (cut_k && prm.top_k <= kListK && sum > 1e-10f) {
            const unsigned T = list_bound(top, prm.top_k);
            if (__float_as_uint(top) >= T)
                for (int i = tid; i < V; i += ST)
                    if (__float_as_uint(w[i]) >= T) {
                        const int q = atomicAdd(&listed, 1);
                        if (q < kList) { lv[q] = w[i]; li[q] = i; }
                    }
            __syncthreads();
            n_list = listed;
        }
        if (!(sum > 1e-10f)) {
            // degenerate mass: uniform fallback (sampling.rs:160-167)
            if (tid == 0) found = (int)(next_u64(rng_state) % (unsigned long long)V);
            __syncthreads();
            token = found;
        } else if (n_list <= kList) {
            token = draw_from_list(n_list, sum, prm, lv, li, lsv, lsi, red, rng_state);
        } else {
            for (int i = tid; i < V; i += ST) w[i] /= sum;
            __syncthreads();
            // 3. top-k: the k-th largest probability by bisection on its bit pattern
            if (cut_k) {
                unsigned T = 0;
                for (int bit = 30; bit >= 0; --bit) {
                    const unsigned cand = T | (1u << bit);
                    int c = 0;
                    for (int i = tid; i < V; i += ST) c += __float_as_uint(w[i]) >= cand;
                    if (bsum_int(c, red) >= prm.top_k) T = cand;
                }
                const float threshold = __uint_as_float(T);
                for (int i = tid; i < V; i += ST)
                    if (w[i] < threshold) w[i] = 0.0f;
                __syncthreads();
            }
            // 4. top-p: the largest cut whose kept mass still reaches top_p
            if (prm.top_p < 1.0f) {
                unsigned T = 0;
                for (int bit = 30; bit >= 0; --bit) {
                    const unsigned cand = T | (1u << bit);
                    float m = 0.0f;
                    for (int i = tid; i < V; i += ST) m += __float_as_uint(w[i]) >= cand ? w[i] : 0.0f;
                    const float kept = bsum(m, red);
                    if (kept >= prm.top_p && kept > 0.0f) T = cand;   // kept > 0: the cut never passes the top token
                }
                // the top token always stays (T never exceeds the maximum that carries mass)
                const float cut = __uint_as_float(T);
                for (int i = tid; i < V; i += ST)
                    if (w[i] < cut) w[i] = 0.0f;
                __syncthreads();
            }
            // 5. renormalise and draw
            float s2 = 0.0f;
            for (int i = tid; i < V; i += ST) s2 += w[i];
            const float sum2 = bsum(s2, red);
            for (int i = tid; i < V; i += ST) w[i] /= sum2;
            if (tid == 0) {
                r_draw = (float)(next_u64(rng_state) >> 40) / 16777216.0f;   // rng.rs:37-40
                found = 0x7fffffff;
            }
            __syncthreads();
            // pick_by_mass (sampling.rs:106-121): thread t owns indices [t*chunk, (t+1)*chunk)
            const int chunk = (V + ST - 1) / ST, i0 = min(tid * chunk, V), i1 = min(i0 + chunk, V);
            float local = 0.0f;
            int last = -1;
            for (int i = i0; i < i1; ++i)
                if (w[i] > 0.0f) { local += w[i]; last = i; }
            // exclusive scan of the chunk masses over the threads
            float incl = local;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float v = __shfl_up_sync(0xffffffffu, incl, o);
                if ((tid & 31) >= o) incl += v;
            }
            if ((tid & 31) == 31) red[tid >> 5] = incl;
            __syncthreads();
            float base = incl - local;
            for (int q = 0; q < (tid >> 5); ++q) base += red[q];
            const float r = r_draw;
            float cum = base;
            for (int i = i0; i < i1; ++i)
                if (w[i] > 0.0f) {
                    cum += w[i];
                    if (r <= cum) { atomicMin(&found, i); break; }
                }
            __syncthreads();
            if (found == 0x7fffffff) {
                // rounding left the total a hair under r: the last index that has any mass
                __shared__ int lasts[ST / 32];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) last = max(last, __shfl_xor_sync(0xffffffffu, last, o));
                if ((tid & 31) == 0) lasts[tid >> 5] = last;
                __syncthreads();
                int l = 0;
                for (int q = 0; q < ST / 32; ++q) l = max(l, lasts[q]);
                token = l;
            } else {
                token = found;
            }
        }
    }
    return token;
}

// The drawn id: to *token_out and, when `state` is given, through the EOS check into queue[tail]. One thread.
__device__ void leave(int token, int* queue, int queue_cap, StepState* state, int* token_out) {
    if (token_out) *token_out = token;
    if (state) {
        if (token == state->eos) {
            state->done = 1;
        } else if (state->tail < queue_cap) {
            queue[state->tail] = token;
            state->tail += 1;
        } else {
            state->error = FC_E_DIM;
        }
    }
}
}  // namespace

// logits_or_probs: V values; from_probs != 0: they are probabilities and the logits are
// ln(max(p, 1e-12)). recent[0 .. n_recent): the ids of the current window.
__global__ void __launch_bounds__(ST, 1)
sample_kernel(const float* __restrict__ in, int V, int from_probs, fc_sampling prm, const int* __restrict__ recent,
              int n_recent_fixed, unsigned long long* rng_state, int* queue, int queue_cap, StepState* state, int* token_out) {
    extern __shared__ __align__(16) float w[];       // [V]
    __shared__ float red[ST / 32];
    __shared__ Lists lists;
    if (state && (state->done | state->error)) return;
    const int token = sample_row(in, V, from_probs, prm, recent, state ? state->tail : n_recent_fixed, rng_state, w, lists, red);
    if (threadIdx.x == 0) leave(token, queue, queue_cap, state, token_out);
}

// The same draw by a cluster of kCluster CTAs, for rows whose top-k takes the list. The passes over the row are bound by what one SM
// issues (a logarithm, a division and an exponential a value; V = 50257, top-k 40, top-p 0.95, 150 penalised ids: 24.9 us, here 16.2); each CTA makes them for the columns
// [rank * COLS, ..) of the row seen as lines of ST values, and only maxima, partial sums and candidates cross between CTAs. A column
// is added from top to bottom and the columns as sample_row's threads are, so that the sum is the same to the bit. A row whose
// mass degenerates or whose ties overflow the list is drawn by rank 0 alone, from the start.
__global__ void __cluster_dims__(kCluster) __launch_bounds__(ST, 1)
sample_cluster_kernel(const float* __restrict__ in, int V, int from_probs, fc_sampling prm, const int* __restrict__ recent,
                      int n_recent_fixed, unsigned long long* rng_state, int* queue, int queue_cap, StepState* state, int* token_out) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) float w[];       // [lines][COLS]; rank 0 alone: [V]
    __shared__ float red[ST / 32], sums[ST / 32], peaks[kCluster], tops[ST];
    __shared__ Lists lists;
    __shared__ int listed, mine, base;
    constexpr int COLS = ST / kCluster, PER = (kSampleMax / ST + kCluster - 1) / kCluster;
    cg::cluster_group all = cg::this_cluster();
    const int rank = all.block_rank(), tid = threadIdx.x, c = tid % COLS, line = tid / COLS, col = rank * COLS + c;
    if (tid == 0) listed = mine = 0;
    all.barrier_arrive();                            // a CTA's shared memory may be written once all have started
    const bool idle = state && (state->done | state->error);   // read by all before rank 0 writes it: the barriers lie between
    const int n_recent = state ? state->tail : n_recent_fixed;
    if (idle) { all.barrier_wait(); return; }
    const int lines = col < V ? (V - 1 - col) / ST + 1 : 0;
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int l = line + kCluster * u;
        if (l < lines) w[l * COLS + c] = logit_of(in[l * ST + col], from_probs);
    }
    __syncthreads();
    penalise(w, V, prm.repetition_penalty, recent, n_recent, lists.at,
             [&](int id) { return id % ST / COLS == rank ? id / ST * COLS + id % COLS : -1; });
    // 2. temperature softmax
    float mx = -INFINITY;
#pragma unroll
    for (int u = 0; u < PER; ++u)
        if (line + kCluster * u < lines) mx = fmaxf(mx, w[(line + kCluster * u) * COLS + c]);
    mx = bmax(mx, red);
    all.barrier_wait();
    if (tid < kCluster) *all.map_shared_rank(peaks + rank, tid) = mx;
    all.sync();
#pragma unroll
    for (int q = 0; q < kCluster; ++q) mx = fmaxf(mx, peaks[q]);
    const float t = fmaxf(prm.temperature, 0.01f);
#pragma unroll
    for (int u = 0; u < PER; ++u) {
        const int l = line + kCluster * u;
        if (l < lines) w[l * COLS + c] = expf((w[l * COLS + c] - mx) / t);
    }
    __syncthreads();
    if (tid < COLS) {
        float s = 0.0f, top = 0.0f;
#pragma unroll 8
        for (int l = 0; l < lines; ++l) {
            const float e = w[l * COLS + c];
            s += e;
            top = fmaxf(top, e);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
#pragma unroll
        for (int q = 0; q < kCluster; ++q) *all.map_shared_rank(tops + col, q) = top;
        if ((tid & 31) < kCluster) *all.map_shared_rank(sums + col / 32, tid & 31) = s;
    }
    all.sync();
    float sum = 0.0f;
#pragma unroll
    for (int q = 0; q < ST / 32; ++q) sum += sums[q];
    const bool mass = sum > 1e-10f;
    if (mass) {
        const unsigned T = list_bound(tops[tid], prm.top_k);
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int l = line + kCluster * u;
            if (l < lines && __float_as_uint(w[l * COLS + c]) >= T) {
                const int q = atomicAdd(&mine, 1);
                if (q < kList) { lists.sv[q] = w[l * COLS + c]; lists.si[q] = l * ST + col; }
            }
        }
        __syncthreads();
        if (tid == 0) base = atomicAdd(all.map_shared_rank(&listed, 0), mine);
        __syncthreads();
        if (tid < mine && base + tid < kList) {
            *all.map_shared_rank(lists.v + base + tid, 0) = lists.sv[tid];
            *all.map_shared_rank(lists.at + base + tid, 0) = lists.si[tid];
        }
        all.sync();
    }
    if (rank) return;
    const int n = listed;
    const int token = mass && n <= kList ? draw_from_list(n, sum, prm, lists.v, lists.at, lists.sv, lists.si, red, rng_state)
                                         : sample_row(in, V, from_probs, prm, recent, n_recent, rng_state, w, lists, red);
    if (tid == 0) leave(token, queue, queue_cap, state, token_out);
}

int launch_sample(const float* in, int V, int from_probs, const fc_sampling& prm, const int* recent, int n_recent,
                  unsigned long long* rng_state, int* queue, int queue_cap, StepState* state, int* token_out, cudaStream_t st) {
    if (V <= 0 || V > kSampleMax) return fail(FC_E_SHAPE, "the device sampler holds a row of at most %d logits in shared memory (V = %d)", kSampleMax, V);
    const size_t smem = (size_t)V * sizeof(float);
    static bool attr_set[64] = {};
    int dev = 0;
    FC_CUDA(cudaGetDevice(&dev));
    if (dev < 64 && !attr_set[dev]) {
        FC_CUDA(cudaFuncSetAttribute(sample_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSampleMax * (int)sizeof(float)));
        FC_CUDA(cudaFuncSetAttribute(sample_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSampleMax * (int)sizeof(float)));
        attr_set[dev] = true;
    }
    // Eight CTAs where the passes over the row outweigh the three exchanges (top-k 40, one CTA / eight: 4096 values 12.7 / 13.6 us,
    // 8192 13.6 / 13.6, 16384 15.9 / 14.5, 50257 24.9 / 16.2), and only for the draws that work on the list: the others would gather the row again.
    if (prm.temperature > 0.0f && prm.top_k > 0 && prm.top_k <= kListK && prm.top_k < V && V >= kClusterRow)
        sample_cluster_kernel<<<kCluster, ST, smem, st>>>(in, V, from_probs, prm, recent, n_recent, rng_state, queue, queue_cap, state, token_out);
    else
        sample_kernel<<<1, ST, smem, st>>>(in, V, from_probs, prm, recent, n_recent, rng_state, queue, queue_cap, state, token_out);
    FC_LAUNCHED();
    return FC_OK;
}

}  // namespace fc
