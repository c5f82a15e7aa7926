// A block of a decode step in two launches: layer/transformer.rs:221-294 (GPT-2) and llm.rs:258-428 (Llama) for one token.
//
//     attention half   x = x0 + (parts + bias); q | k | v = Wqkv LN1(x) + b; append k, v; att = softmax(q Kᵀ / sqrt(hd)) V;
//                      parts_a[h] = Wo[:, head h] att_h                               one cluster of CTAs a head
//     MLP half         x = x0 + (parts_a + bias); hid = gelu(Wup LN2(x) + b) or silu(Wgate RMS(x)) Wup RMS(x);
//                      parts_m[c] = Wdown[:, slice c] hid_c                           one cluster of CTAs a slice of the hidden units
//
// One launch per operation (five a block) costs 16 us a block of width 768, of which the bytes explain 2: each launch pays its
// boundary, an L2 round trip for the row, and the wait of all CTAs for the slowest. What makes two enough is the cluster: the
// q, k and v rows of a head, the parts of its attention and a slice's hidden units travel through distributed shared memory,
// and the product behind them takes the COLUMNS that belong to the head or slice, so that its sums over heads or slices are all that is
// left to the next launch. A cluster reads the row together: each CTA adds up its share of the columns (12 or 16 rows of d floats, from
// L2) and sends it to the others with its mean and squares, from which every CTA makes the norm. (With every CTA reading all of
// it, 50 KB, the row took 4000 cycles from the wait to the norm.)
//
// What CTAs send each other goes by st.async, which counts its bytes on an mbarrier of the receiver: one way, where stores and
// a cluster barrier cost 900 to 1600 cycles. Every wait is bounded; one that runs out raises the status word, and the CTA stays until its
// cluster is through, since its shared memory may yet be written.
//
// Everything that depends on no earlier launch is asked for before the wait: the weights of a CTA's rows and columns (rows in
// registers, a row's levels over the lanes of a warp; columns in registers or, where there are more, in shared memory), norm
// parameters, biases, the cached rows of K and V (cp.async). Sums have a fixed order. A step that is done or failed writes nothing.
// Bound: latency.
#include <algorithm>
#include <atomic>

#include "llama_ops.cuh"
#include "pdl.cuh"

namespace fc {

namespace {

constexpr int T = 384, W = T / 32;             // threads and warps of a CTA (512 with a row of 1024: 339 us a token, 384 317)
constexpr int MAX_D = 1024;
constexpr int MAX_PARTS = 16;
constexpr int MAX_SLICE = 512;                 // hidden units of a cluster
constexpr int MAX_C = 8;

// Two neighbouring levels (bytes B, B + 1 of a word, biased) times two values: packed, half the instructions of one at a time. A byte
// in the mantissa of 2^23 is that plus the byte; less 2^23 + 128 it is the level, exactly.
template <int B>
__device__ __forceinline__ void fma_pair(uint64_t& acc, uint32_t w, uint64_t x) {
    const uint32_t a = __byte_perm(w, 0x4B000000u, 0x7540 + B), b = __byte_perm(w, 0x4B000000u, 0x7541 + B);
    uint64_t v = (uint64_t)b << 32 | a;
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(0xCB000080CB000080ull));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(v));
}
__device__ __forceinline__ float both(uint64_t v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }
// 8 levels against two units of four values.
__device__ __forceinline__ void fma8(uint64_t& acc, uint32_t w0, uint32_t w1, const ulonglong2& x0, const ulonglong2& x1) {
    fma_pair<0>(acc, w0, x0.x);
    fma_pair<2>(acc, w0, x0.y);
    fma_pair<0>(acc, w1, x1.x);
    fma_pair<2>(acc, w1, x1.y);
}
__device__ __forceinline__ float dot16(const uint4& w, const ulonglong2 (&v)[4]) {
    uint64_t s = 0, t = 0;
    fma8(s, w.x, w.y, v[0], v[1]);
    fma8(t, w.z, w.w, v[2], v[3]);
    return both(s) + both(t);
}
__device__ __forceinline__ float dot4(const float4& a, const float4& b, float t) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, t))));
}
__device__ __forceinline__ float warp_sum(float t) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}
__device__ __forceinline__ float4 add4(const float4& a, const float4& b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ uint2 ld_once(const uint2* p) {
    uint2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 ld_once(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t s32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void copy16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s32(dst)), "l"(src) : "memory");
}
// Cluster barrier in two halves; every thread of the cluster takes part in each phase, or has left.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ uint32_t on_rank(const void* p, int rank) {
    uint32_t at;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(s32(p)), "r"(rank));
    return at;
}
// To the same variable of a CTA of the cluster; the bytes count on its barrier.
__device__ __forceinline__ void send(const float* p, const uint64_t* bar, int rank, float v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(on_rank(p, rank)), "f"(v), "r"(on_rank(bar, rank)) : "memory");
}
__device__ __forceinline__ void send(const float2* p, const uint64_t* bar, int rank, float2 v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];"
                 ::"r"(on_rank(p, rank)), "f"(v.x), "f"(v.y), "r"(on_rank(bar, rank)) : "memory");
}
__device__ __forceinline__ void send(const float4* p, const uint64_t* bar, int rank, const float4& v) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(on_rank(p, rank)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(on_rank(bar, rank)) : "memory");
}
// A barrier that one arrival and `bytes` complete, once.
__device__ __forceinline__ void expect(const uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(s32(bar)) : "memory");
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(bar)), "r"(bytes) : "memory");
}
struct Waits {
    int* status;
    StepState* state;                // a wait that runs out fails the step, so that nothing behind it writes or advances
    long long cycles;
    int withhold;                    // test hook: the clusters' first CTAs send nothing of the row (1), no hidden unit (2)
};
__device__ __forceinline__ bool received(const uint64_t* bar, const Waits& w) {
    uint32_t ok;
    auto poll = [&]() {
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], 0;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(s32(bar)) : "memory");
        return ok != 0;
    };
    if (__builtin_expect(poll(), 1)) return true;
    const long long t0 = clock64();
    while (!poll())
        if (clock64() - t0 > w.cycles) {
            if (w.status) atomicExch(w.status, FC_E_TIMEOUT);
            w.state->error = FC_E_TIMEOUT;
            return false;
        }
    return true;
}
// After a wait that ran out: nobody leaves while the cluster may still send to it.
__device__ __forceinline__ void outstay() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    cluster_arrive();
    cluster_wait();
}

// The row a half works on, and its norm.
struct RowIn {
    const float *x, *part, *bias;    // x + (part[0] + .. + part[n_part - 1] + bias); n_part == 0: x
    float* x_out;                    // where the first cluster leaves it (null: nowhere)
    const float *g, *b;
    int n_part, d;
    float eps;
};
// What a model's blocks are made of: LayerNorm, a head of its own for every query, GELU (GPT2); RMSNorm, rotated and grouped heads, SwiGLU
// (LLAMA), the same on matrices of levels alone whose scales belong to the input index (LEVELS): the row is then staged once per
// matrix that reads it, with its scales.
enum Kind { GPT2, LLAMA, LEVELS };

// Staged row: units of 16 bytes; eight consecutive lanes that read two of them each at a stride of 32 bytes meet every bank once.
__device__ __forceinline__ int at16(int i) { return i ^ ((i >> 3) & 1); }

// Shared memory of the row: what arrives (xr, stat, on bar), what is added up (add), the normalised row (xs).
template <int COPIES>
struct RowSmem {
    float4 xr[MAX_D / 4], xs[COPIES][MAX_D / 4], add[W][32];
    float2 stat[MAX_C];
    uint64_t bar;
    __device__ __forceinline__ uint32_t bytes(int d, int C) const { return (uint32_t)(4 * d + 8 * C); }
};
// ahead: what does not depend on the kernel ahead; stage: the normalised row in s.xs, behind two block barriers. A CTA adds at most 32
// units of 16 bytes.
template <int C, bool RMS, int COPIES>
struct RowNormed {
    float4 g, b, pb, scale[COPIES];
    float inv_mine, inv_d;
    __device__ __forceinline__ void ahead(const RowIn& r, int rank, const StepMat* mats) {
        const int tid = threadIdx.x, units = r.d >> 2, mine = units / C;
        inv_d = 1.0f / (float)r.d;
        inv_mine = (float)C * inv_d;
        g = b = pb = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (tid < units) {
            g = ((const float4*)r.g)[tid];
            if (!RMS) b = ((const float4*)r.b)[tid];
            if (COPIES > 1)
#pragma unroll
                for (int i = 0; i < COPIES; ++i) scale[i] = ((const float4*)mats[i].xscale)[tid];
        }
        if (r.n_part && r.bias && tid / 32 < C && (tid & 31) < mine) pb = ((const float4*)r.bias)[rank * mine + (tid & 31)];
    }
    // false: the row never came
    __device__ __forceinline__ bool stage(const RowIn& r, RowSmem<COPIES>& s, int rank, bool first, bool& dead, Waits& waits) {
        const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, units = r.d >> 2, mine = units / C, u = rank * mine + lane;
        // warp w adds rows w - 1 and w - 1 + W; row -1 is x
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        float4 extra = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (r.n_part >= W && wid < C && lane < mine) extra = ((const float4*)r.part)[(size_t)(W - 1) * units + u];   // the row warp 0 leaves out
        if (lane < mine) {
            if (wid == 0) v = ((const float4*)r.x)[u];
            else if (wid <= r.n_part) v = ((const float4*)r.part)[(size_t)(wid - 1) * units + u];
            if (wid + W <= r.n_part) v = wid == 0 ? v : add4(v, ((const float4*)r.part)[(size_t)(wid - 1 + W) * units + u]);
            s.add[wid][lane] = v;
        }
        // behind the row's loads: a branch on them would hold those up for an L2 round trip
        const int error = waits.state->error, done = waits.state->done | error;
        asm volatile("cp.async.wait_all;" ::: "memory");       // every thread's copies are there behind the barrier
        __syncthreads();
        dead = done != 0;
        if (error == FC_E_TIMEOUT) waits.cycles = min(waits.cycles, 10000ll);     // the launches behind a failed one do not wait that long again
        if (wid < C) {
            // warp w sends this CTA's columns to rank w
            float4 t = add4(pb, extra);
#pragma unroll
            for (int i = 1; i < W; ++i) t = add4(t, s.add[i][lane]);            // rows that are not there: zeros
            v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (lane < mine) v = add4(s.add[0][lane], t);
            const float m = RMS ? 0.0f : warp_sum((v.x + v.y) + (v.z + v.w)) * inv_mine;
            float q = 0.0f;
            if (lane < mine) { const float a = v.x - m, c = v.y - m, e = v.z - m, f = v.w - m; q = (a * a + c * c) + (e * e + f * f); }
            q = warp_sum(q);
            if (!(waits.withhold == 1 && rank == 0)) {
                if (lane < mine) send(&s.xr[u], &s.bar, wid, v);
                if (lane == 0) send(&s.stat[rank], &s.bar, wid, make_float2(m, q));
            }
            if (r.x_out && first && wid == 0 && lane < mine && !done) ((float4*)r.x_out)[u] = v;
        }
        // a warp without columns of its own waits at the block barrier instead: one that polls is late to wake, and without a wait it
        // may not read what the peers send
        if (32 * wid >= units) return __syncthreads_and(true);
        const bool ok = received(&s.bar, waits);
        // the CTAs' means and squares are merged around the common mean (n (m - mean)^2 is what a CTA's own mean left out)
        float2 st[C];
#pragma unroll
        for (int i = 0; i < C; ++i) st[i] = s.stat[i];
        float sum = 0.0f, q = 0.0f, dev = 0.0f;
#pragma unroll
        for (int i = 0; i < C; ++i) { sum += st[i].x; q += st[i].y; }
        const float mean = RMS ? 0.0f : sum / (float)C;
        if (!RMS)
#pragma unroll
            for (int i = 0; i < C; ++i) { const float dm = st[i].x - mean; dev = fmaf(dm, dm, dev); }
        const float sd = sqrtf(fmaf(fmaf((float)(4 * mine), dev, q), inv_d, r.eps));
        if (tid < units) {
            float4 x = s.xr[tid];
            if (RMS) {
                const float inv = 1.0f / sd;
                x = make_float4(__fmul_rn(__fmul_rn(x.x, inv), g.x), __fmul_rn(__fmul_rn(x.y, inv), g.y), __fmul_rn(__fmul_rn(x.z, inv), g.z),
                                __fmul_rn(__fmul_rn(x.w, inv), g.w));
            } else {                                           // the reference divides by the deviation
                x = make_float4(((x.x - mean) / sd) * g.x + b.x, ((x.y - mean) / sd) * g.y + b.y, ((x.z - mean) / sd) * g.z + b.z,
                                ((x.w - mean) / sd) * g.w + b.w);
            }
#pragma unroll
            for (int i = 0; i < COPIES; ++i)
                s.xs[i][at16(tid)] = COPIES == 1 ? x : make_float4(x.x * scale[i].x, x.y * scale[i].y, x.z * scale[i].z, x.w * scale[i].w);
        }
        return __syncthreads_and(ok);
    }
};

// RB rows of a matrix against the staged row, by one warp: lanes across k, 8 levels a unit, NU units a lane.
template <int NU, int RB, bool SCALED>
struct WarpRows {
    uint2 q[RB][NU];
    __half d[RB][NU];
    float bias[RB];
    // row r of this matrix becomes the warp's row `slot`
    __device__ __forceinline__ void ahead(int slot, const StepMat& m, int r, int K) {
        const int lane = threadIdx.x & 31, units = K >> 3;
        const size_t at = (size_t)r * m.stride;
        const uint2* src = (const uint2*)(m.qu + at * K);
#pragma unroll
        for (int i = 0; i < NU; ++i) {
            const int u = lane + 32 * i;
            q[slot][i] = u < units ? ld_once(src + u) : make_uint2(0x80808080u, 0x80808080u);
            if (SCALED) d[slot][i] = u < units ? m.d[at * (K >> 5) + (u >> 2)] : __ushort_as_half((unsigned short)0);
        }
        bias[slot] = m.bias ? m.bias[r] : 0.0f;
    }
    // odd_xs: the staged row of rows 1, 3, .. (the two of a SwiGLU pair have matrices of their own)
    __device__ __forceinline__ void run(const float4* xs, const float4* odd_xs, int units, float (&out)[RB]) const {
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int r = 0; r < RB; ++r) out[r] = 0.0f;
#pragma unroll
        for (int i = 0; i < NU; ++i) {
            const int u = lane + 32 * i;
            if (u >= units) break;
            const ulonglong2 x0 = *(const ulonglong2*)&xs[at16(2 * u)], x1 = *(const ulonglong2*)&xs[at16(2 * u + 1)];
            ulonglong2 y0 = x0, y1 = x1;
            if (odd_xs != xs) { y0 = *(const ulonglong2*)&odd_xs[at16(2 * u)]; y1 = *(const ulonglong2*)&odd_xs[at16(2 * u + 1)]; }
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                uint64_t t = 0;
                fma8(t, q[r][i].x, q[r][i].y, r & 1 ? y0 : x0, r & 1 ? y1 : x1);
                out[r] = SCALED ? fmaf(__half2float(d[r][i]), both(t), out[r]) : out[r] + both(t);
            }
        }
#pragma unroll
        for (int r = 0; r < RB; ++r) out[r] = warp_sum(out[r]) + bias[r];
    }
};

struct AttnHalf {
    RowIn in;
    StepMat qkv[3], out;
    StepRope rope;
    float *kc, *vc, *parts;          // parts [heads][d]
    int n_head, n_kv, ctx, cap;      // cap: cached rows a CTA may hold; further ones are read where they are
    Waits waits;
};

// Heads of HD, C = HD / 8 CTAs each, 24 rows of q, k and v a CTA: two for each of the first 12 warps.
template <int HD, int NU, Kind KIND>
__global__ void __launch_bounds__(T, 2) attn_half_kernel(const AttnHalf a) {
    constexpr bool RMS = KIND != GPT2;
    constexpr int COPIES = KIND == LEVELS ? 3 : 1;
    constexpr bool FAR = RMS;                                  // rows beyond the held ones may occur
    constexpr int C = HD / 8, U = HD / 4, KS = HD == 64 ? 80 : HD + 16;   // key rows at a stride of 4 mod 8 units of 16 bytes
    extern __shared__ __align__(16) float sm[];                // K [cap][KS] | V [cap][HD] | scores of the part
    __shared__ __align__(16) RowSmem<COPIES> rs;
    __shared__ __align__(16) float qkv[3][HD], part[W][HD], att[HD], peer_o[C][HD];
    __shared__ float2 peer_ml[C];
    __shared__ float red[2][W];
    __shared__ uint64_t bars[2];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, h = blockIdx.x / C, rank = blockIdx.x % C, d = a.in.d;
    const int kvh = RMS ? h / (a.n_head / a.n_kv) : h, kv_dim = RMS ? a.n_kv * HD : d;
    if (tid == 0) {
        expect(&rs.bar, rs.bytes(d, C));
        expect(&bars[0], 3 * HD * 4);
        expect(&bars[1], C * (HD * 4 + 8));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    cluster_arrive();                                          // a CTA's shared memory may be written once all have started
    // rows i = 2 wid, 2 wid + 1 of this CTA's 24: row rank * 8 + i % 8 of the head's q, k or v
    const bool has_rows = wid < 12;
    const int i0 = 2 * wid;
    WarpRows<NU, 2, KIND != LEVELS> w;
    if (has_rows) {
        const int first = (i0 < 8 ? h : kvh) * HD + rank * 8 + (i0 & 7);
        w.ahead(0, a.qkv[i0 >> 3], first, d);
        w.ahead(1, a.qkv[i0 >> 3], first + 1, d);
    }
    RowNormed<C, RMS, COPIES> row;
    row.ahead(a.in, rank, a.qkv);
    // output rows of this CTA: TPR threads a row, 16 columns each, T / TPR rows a pass
    constexpr int UNITS = HD / 16, TPR = UNITS, PASSES = (MAX_D / C * TPR + T - 1) / T;
    const int per_cta = d / C, sub = tid % TPR, unit = h * UNITS + sub;
    uint4 oq[PASSES];
    float od[PASSES];
#pragma unroll
    for (int i = 0; i < PASSES; ++i) {
        const int n = tid / TPR + i * (T / TPR);
        if (n >= per_cta) continue;
        oq[i] = ld_once((const uint4*)(a.out.qu + (size_t)(rank * per_cta + n) * d) + unit);
        od[i] = KIND == LEVELS ? 1.0f : __half2float(a.out.d[(size_t)(rank * per_cta + n) * (d >> 5) + (unit >> 1)]);
    }
    const float out_scale = KIND == LEVELS && tid < HD ? a.out.xscale[h * HD + tid] : 1.0f;
    // this CTA's part of the positions 0..pos; the last one of the last part is this step's row
    const int pos = a.waits.state->pos, last = min(pos, a.ctx - 1);
    const int per = (int)((unsigned)(last + C) / (unsigned)C), begin = rank * per, len = max(0, min(per, last + 1 - begin));
    const int own = begin + len == last + 1 && len > 0 ? len - 1 : -1;
    float *kt = sm, *vt = sm + (size_t)a.cap * KS, *sc = vt + (size_t)a.cap * HD;
    const float *kg = a.kc + (size_t)begin * kv_dim + (size_t)kvh * HD, *vg = a.vc + (size_t)begin * kv_dim + (size_t)kvh * HD;
    {
        const int held = min(own >= 0 ? own : len, a.cap);
        for (int i = tid; i < held * U; i += T) copy16(kt + (i / U) * KS + (i % U) * 4, kg + (size_t)(i / U) * kv_dim + (i % U) * 4);
        for (int i = tid; i < held * U; i += T) copy16(vt + i * 4, vg + (size_t)(i / U) * kv_dim + (i % U) * 4);
    }
    // threads of the first two warps rotate a pair each, of q, then of k
    const int pair = tid & 31;
    const bool turns = RMS && tid < 64 && pair < a.rope.half;
    float sn = 0.0f, cs = 1.0f;
    if (turns) sincosf(rope_angle(pos, a.rope.ftab[pair], a.rope.inv_linear), &sn, &cs);

    cluster_wait();                                            // all have started
    pdl_wait();
    Waits waits = a.waits;
    bool dead;
    const bool came = row.stage(a.in, rs, rank, blockIdx.x < C, dead, waits);
    pdl_trigger();
    if (!came) { outstay(); return; }
    dead |= pos >= a.ctx;
    if (has_rows) {
        float r[2];
        const float4* xs = rs.xs[COPIES == 1 ? 0 : i0 >> 3];
        w.run(xs, xs, d >> 3, r);
        // every CTA of the cluster gets every row: lane l sends to rank l
        if (lane < C) {
            float* to = &qkv[i0 >> 3][rank * 8 + (i0 & 7)];
            send(to, &bars[0], lane, r[0]);
            send(to + 1, &bars[0], lane, r[1]);
        }
    }
    bool ok = true;
    if (!RMS) {
        ok = received(&bars[0], waits);
    } else {
        if (tid < 64) {
            ok = received(&bars[0], waits);
            if (turns) {
                float* v = qkv[tid >> 5];
                const int i = a.rope.neox ? pair : 2 * pair, j = a.rope.neox ? pair + a.rope.half : i + 1;
                const float x = v[i], y = v[j];
                v[i] = __fsub_rn(__fmul_rn(x, cs), __fmul_rn(y, sn));
                v[j] = __fadd_rn(__fmul_rn(x, sn), __fmul_rn(y, cs));
            }
        }
        ok = __syncthreads_and(ok);
    }
    if (rank == 0 && (!RMS || kvh * (a.n_head / a.n_kv) == h) && tid < 2 * HD && ok && !dead) {
        const int k = tid / HD;
        (k ? a.vc : a.kc)[(size_t)pos * kv_dim + (size_t)kvh * HD + tid % HD] = qkv[1 + k][tid % HD];
    }
    // scores: 4 lanes a key
    const float scale = 1.0f / sqrtf((float)HD);
    const int sl = lane & 3, key0 = wid * 8 + (lane >> 2);
    float4 q[U / 4];
#pragma unroll
    for (int u = 0; u < U / 4; ++u) q[u] = ((const float4*)qkv[0])[u * 4 + sl];
    float top = -INFINITY;
    for (int j0 = 0; j0 < len; j0 += W * 8) {
        const int j = j0 + key0;
        float dot = 0.0f, dot2 = 0.0f;
        if (j < len) {
            auto dots = [&](const float4* k4) {
#pragma unroll
                for (int u = 0; u < U / 4; u += 2) {
                    dot = dot4(q[u], k4[u * 4 + sl], dot);
                    dot2 = dot4(q[u + 1], k4[u * 4 + 4 + sl], dot2);
                }
            };
            // apart, so that the rows in shared memory are read as such
            if (FAR && j >= a.cap && j != own) dots((const float4*)(kg + (size_t)j * kv_dim));
            else dots((const float4*)(j == own ? qkv[1] : kt + j * KS));
        }
        dot += dot2;
        dot += __shfl_xor_sync(0xffffffffu, dot, 1);
        dot += __shfl_xor_sync(0xffffffffu, dot, 2);
        if (j < len) {
            dot *= scale;
            if (sl == 0) sc[j] = dot;
            top = fmaxf(top, dot);
        }
    }
    if (wid * 8 < len) {                                       // the others have no key
#pragma unroll
        for (int o = 16; o > 3; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    }
    if (lane == 0) red[0][wid] = top;
    if (!__syncthreads_and(ok)) { outstay(); return; }
    float M = red[0][0], L = 0.0f;
#pragma unroll
    for (int i = 1; i < W; ++i) M = fmaxf(M, red[0][i]);
    // a part whose scores are all -inf weighs nothing
    const float M0 = M == -INFINITY ? 0.0f : M;
    // P V: U lanes a row
    constexpr int R = T / U;
    const int col = tid % U;
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 2
    for (int j = tid / U; j < len; j += R) {
        float4 v;
        if (FAR && j >= a.cap && j != own) v = ((const float4*)(vg + (size_t)j * kv_dim))[col];
        else v = ((const float4*)(j == own ? qkv[2] : vt + j * HD))[col];
        const float p = expf(sc[j] - M0);
        L += p;
        acc.x = fmaf(p, v.x, acc.x); acc.y = fmaf(p, v.y, acc.y); acc.z = fmaf(p, v.z, acc.z); acc.w = fmaf(p, v.w, acc.w);
    }
#pragma unroll
    for (int o = U; o < 32; o <<= 1) {
        acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
        acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
        acc.z += __shfl_xor_sync(0xffffffffu, acc.z, o);
        acc.w += __shfl_xor_sync(0xffffffffu, acc.w, o);
        L += __shfl_xor_sync(0xffffffffu, L, o);
    }
    if (lane < U) ((float4*)part[wid])[lane] = acc;
    if (lane == 0) red[1][wid] = L;
    __syncthreads();
    if (tid < C * U) {
        // U threads send the part to a rank
        const int to = tid / U;
        float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < W; ++i) o = add4(o, ((const float4*)part[i])[col]);
        L = 0.0f;
#pragma unroll
        for (int i = 0; i < W; ++i) L += red[1][i];
        send(&((const float4*)peer_o[rank])[col], &bars[1], to, o);
        if (col == 0) send(&peer_ml[rank], &bars[1], to, make_float2(M, L));
    }
    ok = true;
    if (tid < HD) {
        ok = received(&bars[1], waits);
        // the parts meet in a fixed order; one without mass weighs nothing
        float2 ml[C];
        float f[C], o[C];
#pragma unroll
        for (int i = 0; i < C; ++i) { ml[i] = peer_ml[i]; o[i] = peer_o[i][tid]; }
#pragma unroll
        for (int i = 0; i < C; ++i) ml[i].x = ml[i].y == 0.0f ? -INFINITY : ml[i].x;
        M = fmaxf(fmaxf(ml[0].x, ml[1 % C].x), fmaxf(ml[2 % C].x, ml[3 % C].x));
#pragma unroll
        for (int i = 4; i < C; ++i) M = fmaxf(M, ml[i].x);
#pragma unroll
        for (int i = 0; i < C; ++i) {
            const float e = expf(ml[i].x - M);
            f[i] = e * ml[i].y;
            o[i] = ml[i].y == 0.0f ? 0.0f : e * o[i];
        }
#pragma unroll
        for (int k = C / 2; k > 0; k >>= 1)
#pragma unroll
            for (int i = 0; i < k; ++i) { f[i] += f[i + k]; o[i] += o[i + k]; }
        att[tid] = KIND == LEVELS ? (o[0] / f[0]) * out_scale : o[0] / f[0];
    }
    if (!__syncthreads_and(ok)) { outstay(); return; }
    ulonglong2 ov[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) ov[j] = ((const ulonglong2*)att)[4 * sub + j];
#pragma unroll
    for (int i = 0; i < PASSES; ++i) {
        const int n = tid / TPR + i * (T / TPR);
        float s = n < per_cta ? od[i] * dot16(oq[i], ov) : 0.0f;
#pragma unroll
        for (int o = TPR >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (n < per_cta && sub == 0 && !dead) a.parts[(size_t)h * d + rank * per_cta + n] = s;
    }
}

struct MlpHalf {
    RowIn in;
    StepMat up[2], down;             // up, or gate and up
    float* parts;                    // [slices][d]
    int slice, F;                    // hidden units of a cluster, of all
    Waits waits;
};

// Clusters of 8; a warp computes RB rows of up (of gate and up in turn: RB / 2 hidden units); 16 threads share RD rows of down, 16 columns of them each: the reads of the hidden units
// from shared memory are what a product of so few columns would else be bound by (with a row a thread 1300 cycles).
template <int NU, int RB, int RD, Kind KIND>
__global__ void __launch_bounds__(T, 2) mlp_half_kernel(const MlpHalf a) {
    constexpr bool RMS = KIND != GPT2;
    constexpr int COPIES = KIND == LEVELS ? 2 : 1, HB = RMS ? RB / 2 : RB;   // HB: hidden units of a warp
    constexpr int C = 8, GROUPS = T / 16;               // RD x GROUPS rows of down: at least d / 8
    extern __shared__ __align__(16) unsigned char cols[];      // this CTA's rows of the slice's columns of down
    __shared__ __align__(16) RowSmem<COPIES> rs;
    __shared__ __align__(16) float hid[MAX_SLICE];
    __shared__ uint64_t bar;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, c = blockIdx.x / C, rank = blockIdx.x % C, d = a.in.d;
    if (tid == 0) {
        expect(&rs.bar, rs.bytes(d, C));
        expect(&bar, a.slice * 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    cluster_arrive();
    const int share = a.slice / C, u0 = wid * HB;              // this warp's first unit of the CTA's share
    WarpRows<NU, RB, KIND != LEVELS> w;
    float down_scale[HB];
#pragma unroll
    for (int i = 0; i < HB; ++i) {
        const int f = c * a.slice + rank * share + min(u0 + i, share - 1);
        if (RMS) {
            w.ahead(2 * i, a.up[0], f, d);
            w.ahead(2 * i + 1, a.up[1], f, d);
        } else {
            w.ahead(i, a.up[0], f, d);
        }
        down_scale[i] = KIND == LEVELS ? a.down.xscale[f] : 1.0f;
    }
    RowNormed<C, RMS, COPIES> row;
    row.ahead(a.in, rank, a.up);
    const int per_cta = d / C, units = a.slice >> 4, unit = tid & 15;
    for (int i = tid; i < per_cta * units; i += T) {
        const int n = i / units, u = i % units;
        copy16(cols + i * 16, a.down.qu + (size_t)(rank * per_cta + n) * a.F + c * a.slice + u * 16);
    }
    float dd[RD];
#pragma unroll
    for (int i = 0; i < RD; ++i) {
        const int n = tid / 16 + i * GROUPS;
        dd[i] = KIND == LEVELS ? 1.0f
              : n < per_cta && unit < units ? __half2float(a.down.d[(size_t)(rank * per_cta + n) * (a.F >> 5) + ((c * units + unit) >> 1)]) : 0.0f;
    }

    cluster_wait();                                            // all have started
    pdl_wait();
    Waits waits = a.waits;
    bool dead;
    const bool came = row.stage(a.in, rs, rank, blockIdx.x < C, dead, waits);
    pdl_trigger();
    if (!came) { outstay(); return; }
    float r[RB];
    w.run(rs.xs[0], rs.xs[COPIES - 1], d >> 3, r);
#pragma unroll
    for (int i = 0; i < HB; ++i)
        if (lane < C && u0 + i < share && !(waits.withhold == 2 && rank == 0)) {
            const int e = rank * share + u0 + i;
            float v;
            if constexpr (RMS) v = __fmul_rn(__fdiv_rn(r[2 * i], __fadd_rn(1.0f, expf(-r[2 * i]))), r[2 * i + 1]);
            else v = gelu_f(r[i]);
            send(&hid[e ^ ((e >> 3) & 12)], &bar, lane, KIND == LEVELS ? v * down_scale[i] : v);
        }
    // a warp goes on, or gives up, as a whole: what follows exchanges among its lanes, and nothing among warps
    if (!__all_sync(0xffffffffu, received(&bar, waits))) { outstay(); return; }
    // eight threads that read the same quarter of their units meet every bank once: quarter j of unit u lies at j ^ (u / 2) % 4
    ulonglong2 v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = ((const ulonglong2*)hid)[4 * unit + (j ^ ((unit >> 1) & 3))];
    float s[8] = {};
#pragma unroll
    for (int i = 0; i < RD; ++i) {
        const int n = tid / 16 + i * GROUPS;
        const bool have = n < per_cta && unit < units;
        const float t = dd[i] * dot16(((const uint4*)cols)[have ? n * units + unit : 0], v);
        s[i] = have ? t : 0.0f;
    }
    // transposing sum over the 16 threads: of four rows, threads 4 j to 4 j + 3 end up with row j, of eight, threads 2 j and 2 j + 1
    constexpr int R = RD <= 4 ? 4 : 8, PER = 16 / R;
#pragma unroll
    for (int o = 8, m = R / 2; m > 0; o >>= 1, m >>= 1) {
        const bool up = unit & o;
#pragma unroll
        for (int i = 0; i < m; ++i) {
            const float keep = up ? s[i + m] : s[i], give = up ? s[i] : s[i + m];
            s[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
#pragma unroll
    for (int o = PER / 2; o > 0; o >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
    const int n = tid / 16 + unit / PER * GROUPS;
    if (unit % PER == 0 && unit / PER < RD && n < per_cta && !dead) a.parts[(size_t)c * d + rank * per_cta + n] = s[0];
}

template <class K, class A>
int launch_clusters(K kernel, int grid, int cluster, size_t smem, cudaStream_t st, const A& a) {
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(T);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    FC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024));
    FC_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
    ++g_launches;
    return FC_OK;
}

// Clusters that share the hidden units: as many as leave a warp two or three rows of up, or of gate and up two or four.
int mlp_slices(int F, bool gated) {
    for (int n : {16, 8, 4, 2, 1}) {
        const int share = F / (n * 8), per_warp = (share + W - 1) / W;
        if (F % (n * 8) == 0 && F / n % 32 == 0 && F / n <= 256 && per_warp <= (gated ? 2 : 3) && per_warp >= (gated ? 1 : 2)) return n;
    }
    return 0;
}
constexpr int HELD = 128;      // cached rows a CTA holds: two CTAs an SM
int attn_cap(int ctx) { return std::min(HELD, (ctx + 7) / 8); }
size_t attn_half_smem(int ctx) { return ((size_t)attn_cap(ctx) * (80 + 64) + (size_t)((ctx + 7) / 8)) * 4; }

}  // namespace

// Heads of 64 (8 CTAs each), rows of 512 to 1024 in multiples of 128, hidden units that split evenly. Us a token on two launches a block (on
// five): 12 x 768 at 32 positions 140 (217), at 256 142 (237), at 900 153 (255); 24 x 1024 317 (447), 322 (488), 339 (533); Llama, 16 x 512, int8 levels, 33 + 64 tokens 12.8 ms (17.3). Narrower rows keep a
// launch per operation, which is what a step of 128 columns is counted in.
bool block_step_covers(int d, int n_head, int F, int ctx, bool gated) {
    return d % 128 == 0 && d >= 512 && d <= MAX_D && n_head * 64 == d && n_head <= MAX_PARTS && mlp_slices(F, gated) > 0 &&
           (gated ? attn_half_smem(ctx) <= 90 * 1024 : ctx <= 8 * HELD);
}
int block_step_slices(int F, bool gated) { return mlp_slices(F, gated); }

int launch_attn_half(const BlockRow& r, int n_head, int n_kv, const StepRope& rope, const StepMat (&qkv)[3], const StepMat& out, float* kc, float* vc, int ctx,
                     float* parts, StepState* state, int* status, cudaStream_t st) {
    constexpr int HD = 64, C = HD / 8;
    const int d = r.d;
    const AttnHalf a = {{r.x, r.part, r.bias, r.x_out, r.g, r.b, r.n_part, d, r.eps}, {qkv[0], qkv[1], qkv[2]}, out, rope, kc, vc, parts, n_head, n_kv, ctx,
                        attn_cap(ctx), {status, state, g_debug.wait_cycles, g_debug.withhold}};
    auto go = [&](auto kernel) { return launch_clusters(kernel, n_head * C, C, attn_half_smem(ctx), st, a); };
    auto of = [&](auto kind) {
        constexpr Kind K = decltype(kind)::value;
        return d > 768 ? go(attn_half_kernel<HD, 4, K>) : d > 512 ? go(attn_half_kernel<HD, 3, K>) : go(attn_half_kernel<HD, 2, K>);
    };
    if (r.b) return of(std::integral_constant<Kind, GPT2>());
    return out.xscale ? of(std::integral_constant<Kind, LEVELS>()) : of(std::integral_constant<Kind, LLAMA>());
}

int launch_mlp_half(const BlockRow& r, const StepMat (&up)[2], const StepMat& down, int F, float* parts, StepState* state, int* status, cudaStream_t st) {
    const bool gated = !r.b;
    const int d = r.d, slices = mlp_slices(F, gated), slice = F / slices, per_warp = (slice / 8 + W - 1) / W;
    const MlpHalf a = {{r.x, r.part, r.bias, r.x_out, r.g, r.b, r.n_part, d, r.eps}, {up[0], up[1]}, down, parts, slice, F,
                       {status, state, g_debug.wait_cycles, g_debug.withhold}};
    auto go = [&](auto kernel) { return launch_clusters(kernel, slices * 8, 8, (size_t)(d / 8) * slice, st, a); };
    // FEW, MANY: rows of a warp
    auto of = [&](auto kind, auto few, auto many) {
        constexpr Kind K = decltype(kind)::value;
        constexpr int FEW = decltype(few)::value, MANY = decltype(many)::value;
        const bool more = per_warp * (gated ? 2 : 1) > FEW;
        if (d > 768) return more ? go(mlp_half_kernel<4, MANY, 6, K>) : go(mlp_half_kernel<4, FEW, 6, K>);
        if (d > 512) return more ? go(mlp_half_kernel<3, MANY, 4, K>) : go(mlp_half_kernel<3, FEW, 4, K>);
        return more ? go(mlp_half_kernel<2, MANY, 4, K>) : go(mlp_half_kernel<2, FEW, 4, K>);
    };
    const std::integral_constant<int, 2> two;
    const std::integral_constant<int, 3> three;
    const std::integral_constant<int, 4> four;
    if (!gated) return of(std::integral_constant<Kind, GPT2>(), two, three);
    return down.xscale ? of(std::integral_constant<Kind, LEVELS>(), two, four) : of(std::integral_constant<Kind, LLAMA>(), two, four);
}

}  // namespace fc
