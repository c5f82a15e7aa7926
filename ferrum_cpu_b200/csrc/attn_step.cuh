// One attention step of a decode chain: rotate q and k (or take them as they are), append k and v to the caches, and the
// single-query softmax over positions 0..pos — AttentionHead::forward_cached (attention.rs:140-196) and its grouped-query form
// (llm.rs:258-349) — one CTA per query head, or at long positions a cluster of them, each with a part of the positions, whose
// outputs meet in the first one's shared memory in rank order.
//
// A step of some hundred positions is bound by latency: a head reads 2 * 4 * hd bytes a position, 50 KB at hd 64 and 100
// positions, but from L2 or DRAM, behind a chain of dependent reads (state, q row, keys, scores, values). So everything that
// earlier steps wrote — the state and the cached rows of K and V — is asked for before the wait on the qkv product (cp.async
// into shared memory), and after the wait only this step's q, k and v are missing. Keys are stored at a stride of 4 mod 8
// units of 16 bytes, so that the 4 lanes that share a key and the 8 keys of a warp's sweep read every bank once; values are
// read row by row and need no padding. Rows that do not fit in shared memory are read where they are: at 37 ns a row and head
// (64 wide) against 12 ns for a held one, which is why a head that long is shared.
// 256 threads, and q, k and v asked for ahead of the check of the state: a step of 12 layers of width 768 takes 226.6 us; with
// 512 threads and the loads behind the check 232.6 us.
//
// The two forms are instances in files of their own (attn_step.cu, attn_step_split.cu): their images are loaded apart. With both in
// one, the one-CTA steps of a model that streams more than the L2 holds lost 0.9 % (16 blocks, 2048 wide, 64 tokens: 43.62 ms; 43.25
// apart).
#pragma once
#include <algorithm>
#include <atomic>

#include "llama_ops.cuh"
#include "pdl.cuh"

namespace fc {

struct AttnStep {
    const float* qkv;
    int n_q, n_kv, half, neox;
    const float2* ftab;
    float inv_linear;
    float *kc, *vc;
    int ctx, split;
};
int launch_attn_step_split(int hd, const AttnStep& a, const StepState* state, float* out, cudaStream_t st);

namespace {

constexpr int THREADS = 256, WARPS = THREADS / 32;
constexpr size_t kSmem = 204 * 1024;
constexpr int MAX_SPLIT = 8, MIN_SPLIT = 4;   // CTAs that share a head (of two or three, no shape was at hand to measure)
constexpr int PART = 64;                      // positions for which another of them takes part

template <int HD>
struct KStride { static constexpr int v = HD == 64 ? 80 : HD + 16; };     // floats: 48, 80, 144

__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ float dot4(const float4& a, const float4& b, float t) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, t))));
}

// Cluster barrier in two halves; every thread of the cluster takes part in each phase.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// To the same variable of rank 0 of the cluster.
__device__ __forceinline__ void store_rank0(float* p, float v) {
    uint32_t at;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(at) : "r"((uint32_t)__cvta_generic_to_shared(p)));
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(at), "f"(v) : "memory");
}

template <int HD, bool SPLIT>
__global__ void __launch_bounds__(THREADS, 1) attn_step_kernel(const float* __restrict__ qkv, int n_q, int n_kv, int half, int neox,
                                                               const float2* __restrict__ ftab, float inv_linear, float* kc, float* vc,
                                                               int ctx, int n_split, int cap, const StepState* st, float* __restrict__ out) {
    constexpr int KS = KStride<HD>::v, U = HD / 4;            // units of 16 bytes in a row
    extern __shared__ __align__(16) float sm[];               // K [cap][KS] | V [cap][HD] | scores [positions of a part]
    __shared__ __align__(16) float qs[HD], ks[HD], vs[HD];
    __shared__ __align__(16) float part[WARPS][HD];
    __shared__ float red[2][WARPS];
    __shared__ float peer_o[MAX_SPLIT][HD], peer_ml[MAX_SPLIT][2];   // rank 0: each part's output, largest score and mass
    const int split = SPLIT ? n_split : 1;
    if (SPLIT) cluster_arrive();                              // a CTA's shared memory may be written once all have started
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int h = SPLIT ? blockIdx.x / split : blockIdx.x, rank = SPLIT ? blockIdx.x - h * split : 0, group = n_q / n_kv, kvh = h / group, kv_dim = n_kv * HD;
    const int pos = st->pos;
    // this CTA's part of the positions 0..pos: from `begin` on, `len` of them; the last one of the last part is this step's row
    const int parts = SPLIT ? min(split, pos / PART + 1) : 1, per = SPLIT ? (int)((unsigned)(pos + parts) / (unsigned)parts) : pos + 1;
    const int begin = rank * per, len = !SPLIT ? pos + 1 : rank < parts ? min(per, pos + 1 - begin) : 0;
    const int own = !SPLIT ? pos : rank == parts - 1 ? len - 1 : -1;
    const bool owner = !SPLIT || own >= 0;
    float *kt = sm, *vt = sm + (size_t)cap * KS, *sc = vt + (size_t)cap * HD;
    const float *kg = kc + (size_t)begin * kv_dim + (size_t)kvh * HD, *vg = vc + (size_t)begin * kv_dim + (size_t)kvh * HD;
    const int held = min(owner ? own : len, cap);
    for (int i = tid; i < held * U; i += THREADS) copy16(kt + (i / U) * KS + (i % U) * 4, kg + (size_t)(i / U) * kv_dim + (i % U) * 4);
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int i = tid; i < held * U; i += THREADS) copy16(vt + i * 4, vg + (size_t)(i / U) * kv_dim + (i % U) * 4);
    asm volatile("cp.async.commit_group;" ::: "memory");
    // HD threads each build q and k (rotated pairs, then the unrotated tail) and hold v; with 2 HD threads q and k, then v
    constexpr int ROLES = THREADS / HD < 3 ? 2 : 3;
    const int role = tid / HD, t = tid % HD;
    const bool pair = role < 2 && t < half, plain = role == 2 || (role < 2 && t >= 2 * half);
    float s = 0.0f, c = 1.0f;
    if (pair) sincosf(rope_angle(pos, ftab[t], inv_linear), &s, &c);

    pdl_wait();
    pdl_trigger();       // not ahead of the wait: what the kernel behind asks for would queue up before this one's row
    // asked for ahead of the check of the state, which is as far away
    const float* src = qkv + (role == 0 ? (size_t)h * HD : (size_t)n_q * HD + (size_t)(role == 2) * kv_dim + (size_t)kvh * HD);
    const int ia = pair ? (neox ? t : 2 * t) : t, ib = neox ? t + half : 2 * t + 1;
    float a = 0.0f, b = 0.0f, v_own = 0.0f;
    if (pair | plain) a = src[ia];
    if (pair) b = src[ib];
    if (ROLES == 2 && role == 0) v_own = qkv[(size_t)n_q * HD + kv_dim + (size_t)kvh * HD + t];
    if ((st->done | st->error) || pos >= ctx || (rank > 0 && parts == 1)) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (SPLIT) cluster_wait();
        return;
    }
    float* dst = role == 0 ? qs : role == 1 ? ks : vs;
    if (pair) {
        dst[ia] = __fsub_rn(__fmul_rn(a, c), __fmul_rn(b, s));
        dst[ib] = __fadd_rn(__fmul_rn(a, s), __fmul_rn(b, c));
    } else if (plain) {
        dst[t] = a;
    }
    if (ROLES == 2 && role == 0) vs[t] = v_own;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    if (h == kvh * group && owner && tid < 2 * HD) {
        float* row = (role ? vc : kc) + (size_t)pos * kv_dim + (size_t)kvh * HD;
        row[t] = role ? vs[t] : ks[t];
    }
    // scores: 4 lanes a key
    const float scale = 1.0f / sqrtf((float)HD);
    const int sub = lane & 3, key0 = wid * 8 + (lane >> 2);
    const float4* q4 = (const float4*)qs;
    float4 q[U / 4];
#pragma unroll
    for (int u = 0; u < U / 4; ++u) q[u] = q4[u * 4 + sub];
    float top = -INFINITY, mass = 0.0f;
    for (int j0 = 0; j0 < len; j0 += WARPS * 8) {
        const int j = j0 + key0;
        float dot = 0.0f;
        if (j < len) {
            const float4* k4 = j == own ? (const float4*)ks : j < cap ? (const float4*)(kt + (size_t)j * KS) : (const float4*)(kg + (size_t)j * kv_dim);
#pragma unroll
            for (int u = 0; u < U / 4; ++u) dot = dot4(q[u], k4[u * 4 + sub], dot);
        }
        dot += __shfl_xor_sync(0xffffffffu, dot, 1);
        dot += __shfl_xor_sync(0xffffffffu, dot, 2);
        if (j < len) {
            dot *= scale;
            if (sub == 0) sc[j] = dot;
            if (dot > top) { mass *= expf(top - dot); top = dot; }
            if (dot != -INFINITY) mass += expf(dot - top);
        }
    }
    float wtop = top;
#pragma unroll
    for (int o = 16; o > 3; o >>= 1) wtop = fmaxf(wtop, __shfl_xor_sync(0xffffffffu, wtop, o));
    mass = mass == 0.0f ? 0.0f : mass * expf(top - wtop);
#pragma unroll
    for (int o = 16; o > 3; o >>= 1) mass += __shfl_xor_sync(0xffffffffu, mass, o);
    if (lane == 0) { red[0][wid] = wtop; red[1][wid] = mass; }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    float M = red[0][0], L = 0.0f;
#pragma unroll
    for (int w = 1; w < WARPS; ++w) M = fmaxf(M, red[0][w]);
#pragma unroll
    for (int w = 0; w < WARPS; ++w) L += red[1][w] == 0.0f ? 0.0f : red[1][w] * expf(red[0][w] - M);
    // P V: U lanes a row
    constexpr int R = THREADS / U;
    const int col = tid % U, r0 = tid / U;
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 2
    for (int j = r0; j < len; j += R) {
        const float4* v4 = j == own ? (const float4*)vs : j < cap ? (const float4*)(vt + (size_t)j * HD) : (const float4*)(vg + (size_t)j * kv_dim);
        const float p = expf(sc[j] - M);
        const float4 v = v4[col];
        acc.x = fmaf(p, v.x, acc.x); acc.y = fmaf(p, v.y, acc.y); acc.z = fmaf(p, v.z, acc.z); acc.w = fmaf(p, v.w, acc.w);
    }
#pragma unroll
    for (int o = U; o < 32; o <<= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
        acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
        acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
    }
    if (lane < U) ((float4*)part[wid])[lane] = acc;
    __syncthreads();
    float o = 0.0f;
    if (tid < HD) {
#pragma unroll
        for (int w = 0; w < WARPS; ++w) o += part[w][tid];
        if (parts == 1) out[(size_t)h * HD + tid] = o / L;
    }
    if (!SPLIT) return;
    cluster_wait();
    if (parts == 1) return;
    // the parts meet in rank 0, in rank order
    if (len > 0 && tid < HD) store_rank0(&peer_o[rank][tid], o);
    if (len > 0 && tid < 2) store_rank0(&peer_ml[rank][tid], tid ? L : M);
    cluster_arrive();
    cluster_wait();
    if (rank > 0 || tid >= HD) return;
    M = peer_ml[0][0];
    for (int r = 1; r < parts; ++r) M = fmaxf(M, peer_ml[r][0]);
    L = o = 0.0f;
    for (int r = 0; r < parts; ++r) {
        if (peer_ml[r][1] == 0.0f) continue;                  // nothing in this part weighs anything
        const float w = expf(peer_ml[r][0] - M);
        L = fmaf(w, peer_ml[r][1], L);
        o = fmaf(w, peer_o[r][tid], o);
    }
    out[(size_t)h * HD + tid] = o / L;
}

template <int HD, bool SPLIT>
int prepare() {
    static std::atomic<unsigned long long> ready{0};
    int dev = 0;
    FC_CUDA(cudaGetDevice(&dev));
    if (!(ready.load() >> (dev & 63) & 1)) {
        FC_CUDA(cudaFuncSetAttribute(attn_step_kernel<HD, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem));
        ready.fetch_or(1ull << (dev & 63));
    }
    return FC_OK;
}
// Rows a CTA of a head shared by `split` of them may hold, and its dynamic shared memory.
template <int HD>
void room(int ctx, int split, int* cap, size_t* smem) {
    const int longest = split == 1 ? ctx : std::max(std::min(PART, ctx), (ctx + split - 1) / split);
    const size_t scores = (size_t)longest * 4, row = (KStride<HD>::v + HD) * 4;
    *cap = std::min(longest, (int)((kSmem - scores) / row));
    *smem = *cap * row + scores;
}
template <int HD, bool SPLIT>
int launch(const AttnStep& a, const StepState* state, float* out, cudaStream_t st) {
    int cap = 0;
    size_t smem = 0;
    room<HD>(a.ctx, a.split, &cap, &smem);
    FC_TRY((prepare<HD, SPLIT>()));
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = a.split;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(a.n_q * a.split);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = SPLIT ? 2 : 1;
    FC_CUDA(cudaLaunchKernelEx(&cfg, attn_step_kernel<HD, SPLIT>, a.qkv, a.n_q, a.n_kv, a.half, a.neox, a.ftab, a.inv_linear, a.kc, a.vc, a.ctx,
                               a.split, cap, state, out));
    ++g_launches;
    return FC_OK;
}

}  // namespace
}  // namespace fc
