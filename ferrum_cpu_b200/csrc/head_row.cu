// The LM head of a decode step, behind block_step.cu: logits = Whead LN(x + (parts + bias)), and per CTA the largest logit and the
// mass around it (model.rs:51-71, ops.rs:478-502 for one row).
//
// One row against a matrix of tens of thousands of rows. A lane keeps its share of the normalised row in REGISTERS for all rows of
// its warp (units of 8 levels, NU a lane), so that the loop reads nothing but weights: per pair of levels two byte permutes, a packed
// subtract and a packed multiply-add. Two to four tasks of two rows are in flight a warp, all asked for before the wait: a quarter of the
// matrix is under way when the row appears.
// Bound: HBM and issue.
#include <algorithm>

#include "fc_common.cuh"
#include "pdl.cuh"

namespace fc {

namespace {

constexpr int T = 512, W = T / 32, RB = 2, MAX_PARTS = 16;
static_assert(RB * W == kHeadSpan, "consecutive rows of a CTA");

__device__ __forceinline__ uint64_t pack2(float lo, float hi) { return (uint64_t)__float_as_uint(hi) << 32 | __float_as_uint(lo); }
// Levels 2 i and 2 i + 1 of a unit's word against two elements of the row.
template <int B>
__device__ __forceinline__ void fma_pair(uint64_t& acc, uint32_t w, uint64_t x) {
    const uint32_t a = __byte_perm(w, 0x4B000000u, 0x7540 + B), b = __byte_perm(w, 0x4B000000u, 0x7541 + B);
    uint64_t v = (uint64_t)b << 32 | a;
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(0xCB000080CB000080ull));   // less 2^23 + 128
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(v));
}
__device__ __forceinline__ float warp_sum(float t) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}

struct HeadArgs {
    const uint8_t* qu; const __half* d; int N, K;
    const float *x, *part, *bias, *g, *b, *xscale;
    int n_part;
    float eps;
    float* out; float2* stats;
    const StepState* state;
};

// RMS: RMSNorm in LayerNorm's place. SCALED: f16 scales per 32 of k, else levels alone and the scales of the input indices.
template <int NU, bool RMS, bool SCALED>
__global__ void __launch_bounds__(T, 1) head_row_kernel(const HeadArgs a) {
    constexpr int DEPTH = NU <= 2 ? 4 : NU == 3 ? 3 : 2;     // tasks in flight: as many as the registers hold
    extern __shared__ __align__(16) float4 add[];            // [n_part + 1][K / 4]
    __shared__ float red[2][W];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, K = a.K, units = K >> 3, quads = K >> 2;
    const int tasks = (a.N + RB - 1) / RB, step = gridDim.x * W, first = blockIdx.x * W + wid;
    struct Rows { uint2 q[RB][NU]; __half d[RB][NU]; } w[DEPTH];
    auto fetch = [&](Rows& r, int t) {
        if (t >= tasks) return;
#pragma unroll
        for (int i = 0; i < RB; ++i) {
            const size_t row = (size_t)min(t * RB + i, a.N - 1);
            const uint2* q = (const uint2*)(a.qu + row * K);
            const __half* d = a.d + row * (K >> 5);
#pragma unroll
            for (int u = 0; u < NU; ++u) {
                if (lane + 32 * u >= units) continue;
                asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];" : "=r"(r.q[i][u].x), "=r"(r.q[i][u].y) : "l"(q + lane + 32 * u));
                if (SCALED) r.d[i][u] = d[(lane + 32 * u) >> 2];
            }
        }
    };
#pragma unroll
    for (int i = 0; i < DEPTH; ++i) fetch(w[i], first + i * step);
    float4 g = {}, b = {}, pb = {}, xs = {};
    if (tid < quads) {
        g = ((const float4*)a.g)[tid];
        if (!RMS) b = ((const float4*)a.b)[tid];
        if (!SCALED) xs = ((const float4*)a.xscale)[tid];
        if (a.n_part && a.bias) pb = ((const float4*)a.bias)[tid];
    }

    pdl_wait();
    // the row: a warp brings a part, then a thread adds up four columns
    for (int p = wid; p <= a.n_part; p += W) {
        const float4* src = p == 0 ? (const float4*)a.x : (const float4*)a.part + (size_t)(p - 1) * quads;
        for (int i = lane; i < quads; i += 32) add[p * quads + i] = src[i];
    }
    const bool dead = (a.state->done | a.state->error) != 0;
    __syncthreads();
    pdl_trigger();
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (tid < quads) {
        for (int p = 1; p <= a.n_part; ++p) {
            const float4 t = add[p * quads + tid];
            pb.x += t.x; pb.y += t.y; pb.z += t.z; pb.w += t.w;
        }
        v = add[tid];
        v.x += pb.x; v.y += pb.y; v.z += pb.z; v.w += pb.w;
    }
    // every warp takes the mean of its own elements and the squares around it; merged around the common mean
    auto count = [&](int wi) { return (float)min(max(K - 128 * wi, 0), 128); };
    const float n_w = count(wid), m_w = !RMS && n_w > 0.0f ? warp_sum((v.x + v.y) + (v.z + v.w)) / n_w : 0.0f;
    float q = 0.0f;
    if (tid < quads) { const float e = v.x - m_w, f = v.y - m_w, h = v.z - m_w, k = v.w - m_w; q = (e * e + f * f) + (h * h + k * k); }
    q = warp_sum(q);
    if (lane == 0) { red[0][wid] = m_w; red[1][wid] = q; }
    __syncthreads();
    float mean = 0.0f, m2 = 0.0f;
#pragma unroll
    for (int i = 0; i < W; ++i) mean += count(i) * red[0][i];
    mean = RMS ? 0.0f : mean / (float)K;
#pragma unroll
    for (int i = 0; i < W; ++i) { const float dm = red[0][i] - mean; m2 += fmaf(count(i) * dm, dm, red[1][i]); }
    const float sd = sqrtf(m2 / (float)K + a.eps);
    if (tid < quads) {
        if (RMS) {
            const float inv = 1.0f / sd;
            v = make_float4(__fmul_rn(__fmul_rn(v.x, inv), g.x), __fmul_rn(__fmul_rn(v.y, inv), g.y), __fmul_rn(__fmul_rn(v.z, inv), g.z),
                            __fmul_rn(__fmul_rn(v.w, inv), g.w));
        } else {
            v = make_float4(((v.x - mean) / sd) * g.x + b.x, ((v.y - mean) / sd) * g.y + b.y, ((v.z - mean) / sd) * g.z + b.z, ((v.w - mean) / sd) * g.w + b.w);
        }
        if (!SCALED) { v.x *= xs.x; v.y *= xs.y; v.z *= xs.z; v.w *= xs.w; }
        add[tid] = v;
    }
    __syncthreads();
    uint64_t x[NU][4];
#pragma unroll
    for (int u = 0; u < NU; ++u) {
        float4 lo = {}, hi = {};
        if (lane + 32 * u < units) { lo = add[2 * (lane + 32 * u)]; hi = add[2 * (lane + 32 * u) + 1]; }
        x[u][0] = pack2(lo.x, lo.y); x[u][1] = pack2(lo.z, lo.w); x[u][2] = pack2(hi.x, hi.y); x[u][3] = pack2(hi.z, hi.w);
    }

    float top = -INFINITY, mass = 0.0f;
    auto work = [&](const Rows& r, int t) {
        float s[RB];
#pragma unroll
        for (int i = 0; i < RB; ++i) {
            s[i] = 0.0f;
#pragma unroll
            for (int u = 0; u < NU; ++u) {
                if (lane + 32 * u >= units) continue;
                uint64_t acc = 0;
                fma_pair<0>(acc, r.q[i][u].x, x[u][0]);
                fma_pair<2>(acc, r.q[i][u].x, x[u][1]);
                fma_pair<0>(acc, r.q[i][u].y, x[u][2]);
                fma_pair<2>(acc, r.q[i][u].y, x[u][3]);
                const float t = __uint_as_float((uint32_t)acc) + __uint_as_float((uint32_t)(acc >> 32));
                s[i] = SCALED ? fmaf(__half2float(r.d[i][u]), t, s[i]) : s[i] + t;
            }
        }
        // one value a lane: lanes below 16 end up with row 0, the others with row 1
        float one = lane & 16 ? s[1] : s[0];
        one += __shfl_xor_sync(0xffffffffu, lane & 16 ? s[0] : s[1], 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) one += __shfl_xor_sync(0xffffffffu, one, o);
        const int n = t * RB + (lane >> 4);
        if ((lane & 15) == 0 && n < a.N && !dead) {
            a.out[n] = one;
            if (one > top) { mass *= expf(top - one); top = one; }
            if (one != -INFINITY) mass += expf(one - top);
        }
    };
    for (int t = first; t < tasks; t += DEPTH * step)
#pragma unroll
        for (int i = 0; i < DEPTH; ++i) {
            const int k = t + i * step;
            if (k < tasks) {
                work(w[i], k);
                fetch(w[i], k + DEPTH * step);
            }
        }
    if (!a.stats) return;
    // the two lanes of a warp that finish rows, then the warps
    const float other = __shfl_xor_sync(0xffffffffu, top, 16), m = fmaxf(top, other);
    mass = mass == 0.0f ? 0.0f : mass * expf(top - m);
    mass += __shfl_xor_sync(0xffffffffu, mass, 16);
    __syncthreads();
    if (lane == 0) { red[0][wid] = m; red[1][wid] = mass; }
    __syncthreads();
    if (tid == 0) {
        top = -INFINITY;
        for (int i = 0; i < W; ++i) top = fmaxf(top, red[0][i]);
        mass = 0.0f;
        for (int i = 0; i < W; ++i)
            if (red[1][i] != 0.0f) mass += red[1][i] * expf(red[0][i] - top);
        a.stats[blockIdx.x] = make_float2(top, mass);
    }
}

}  // namespace

int launch_head_row(const StepMat& w, int N, const BlockRow& r, float* logits, float2* stats, int* n_stats, const StepState* state, cudaStream_t st) {
    const int K = r.d;
    if (K % 128 || K > 1024 || r.n_part > MAX_PARTS || (!w.d && (!w.xscale || r.b))) return fail(FC_E_SHAPE, "head row: K = %d, %d rows to add", K, r.n_part);
    static int sms[64] = {};
    int dev = 0;
    FC_CUDA(cudaGetDevice(&dev));
    if (dev >= 64) return fail(FC_E_ARG, "device index %d", dev);
    if (!sms[dev]) FC_CUDA(cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev));
    const HeadArgs a = {w.qu, w.d, N, K, r.x, r.part, r.bias, r.g, r.b, w.xscale, r.n_part, r.eps, logits, stats, state};
    const int blocks = std::min(sms[dev], ((N + RB - 1) / RB + W - 1) / W);
    if (n_stats) *n_stats = blocks;
    const size_t smem = (size_t)(r.n_part + 1) * K * 4;
    auto go = [&](auto kernel) -> int {
        FC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (MAX_PARTS + 1) * 1024 * 4));
        FC_CUDA(launch_pdl(kernel, dim3(blocks), dim3(T), smem, st, a));
        ++g_launches;
        return FC_OK;
    };
    const int nu = (K + 255) / 256;
    auto of = [&](auto rms, auto scaled) {
        constexpr bool R = decltype(rms)::value, S = decltype(scaled)::value;
        return nu == 1 ? go(head_row_kernel<1, R, S>) : nu == 2 ? go(head_row_kernel<2, R, S>) : nu == 3 ? go(head_row_kernel<3, R, S>) : go(head_row_kernel<4, R, S>);
    };
    if (r.b) return of(std::false_type(), std::true_type());
    return w.d ? of(std::true_type(), std::true_type()) : of(std::true_type(), std::false_type());
}

}  // namespace fc
