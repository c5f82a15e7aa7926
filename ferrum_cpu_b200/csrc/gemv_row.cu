// One activation row against quantised matrices: the projections of a decode step and the M = 1 linear.
//
//     y[n] = (residual[n] +) bias[n] + sum_k xhat[k] * w[n][k]
//     xhat = x, RMSNorm(x) (llm.rs:57-64) or LayerNorm(x) (layer/norm.rs:46-82)
//
// Up to three matrices share the row (q | k | v, gate | up). A matrix is a QMat: int8 levels with an f16 scale per 32 of k
// (Q8_0), or levels alone whose scale belongs to the input index (the per-row-scale QWeight of quant.rs:122-146): then
// xhat[k] * scale[k] is staged per matrix (ops.rs:336-342).
//
// A step of a decoder is a chain of such products, each a few microseconds long, so what counts is how little happens
// between "the row is there" and "the result is there":
//  - a warp owns RB rows (or a K slice of them) from the first load to the dot product: lanes across k, 16 levels each. It
//    asks for the first rows BEFORE it waits for the kernel ahead (weights depend on nothing), so small matrices are in
//    registers when the activations appear; the next rows are asked for before the current ones are multiplied;
//  - the norm's parameters, the input scales and, inside a model, the first bias are asked for before that wait too, the first
//    residual (and a caller's bias, which may be what the kernel ahead writes) right after it: later each of them would cost
//    an L2 round trip;
//  - the row is staged in shared memory once, out of registers (two block barriers with a norm, one without; every thread
//    merges the warps' sums itself, over a fixed count with wide reads: with loops over the warps and a division each, 24
//    LayerNorms cost 50 us of a step of width 768, now 27). From there on warps do not meet, unless K is wider than 2048 and
//    `ks` of them share a row;
//  - few rows take few warps per CTA, spread over all SMs.
// Bound: issue and latency. In a chain 768 -> 768 takes 1.8 us, 3072 -> 768 2.8, 2048 -> 2048 3.2, 2048 -> 16384 12.5 (2.8 TB/s;
// 12.4 when the matrix comes from L2), 2048 -> 32000 21; the sum of the launches of a step is what a token costs. (Taken with one level an
// instruction; packed pairs took 5 % off a step of 16 blocks of 2048, 43.1 -> 40.9 ms for 64 tokens. Asking for a warp's second task ahead
// of the wait as well: 43.0.)
// (The kernel this replaced streamed 32 KB tiles through a shared-memory ring with a block barrier per tile: about 5.5 us
// for every product of a step, however small.)
#include <algorithm>
#include <type_traits>

#include "fc_common.cuh"
#include "pdl.cuh"

namespace fc {

namespace {

constexpr int MAX_WARPS = 16;
constexpr int UN = 2;            // 16-byte units of the row a thread stages from registers
constexpr int SLICE = 2048;      // k a warp covers: 4 chunks of 16 per lane

// Two neighbouring quants (bytes B, B + 1 of a word, biased) times two values. A byte in the mantissa of 2^23 is that plus the byte;
// less 2^23 + 128 it is the quant, exactly.
template <int B>
__device__ __forceinline__ void fma_pair(uint64_t& acc, uint32_t w, uint64_t x) {
    const uint32_t a = __byte_perm(w, 0x4B000000u, 0x7540 + B), b = __byte_perm(w, 0x4B000000u, 0x7541 + B);
    uint64_t v = (uint64_t)b << 32 | a;
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(0xCB000080CB000080ull));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(x), "l"(v));
}
__device__ __forceinline__ float both(uint64_t v) { return __uint_as_float((uint32_t)v) + __uint_as_float((uint32_t)(v >> 32)); }
// 16 quants against 16 activations held in registers (shared by the rows of a task), packed: 32 instructions where one at a time
// takes 48.
__device__ __forceinline__ float dot16x(const uint4& w, const ulonglong2& x0, const ulonglong2& x1, const ulonglong2& x2, const ulonglong2& x3) {
    uint64_t a = 0, b = 0;
    fma_pair<0>(a, w.x, x0.x); fma_pair<0>(b, w.z, x2.x);
    fma_pair<2>(a, w.x, x0.y); fma_pair<2>(b, w.z, x2.y);
    fma_pair<0>(a, w.y, x1.x); fma_pair<0>(b, w.w, x3.x);
    fma_pair<2>(a, w.y, x1.y); fma_pair<2>(b, w.w, x3.y);
    return both(a) + both(b);
}
// Levels are read once: they need no place in L1.
__device__ __forceinline__ uint4 ld_levels(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

struct RowArgs {                 // small: a launch costs the host more with every few words of arguments
    GemvPart part[3];
    const float *x, *nw, *nb, *residual;
    const StepState* state;
    float2* stats;               // per CTA: largest output and sum of exp(output - largest), or null
    int K, tasks;
    float eps;
    uint8_t parts, staged;       // staged: copies of the row in shared memory (one per part when the parts have input scales)
    uint8_t ks, epi;             // ks: warps that share a row
};

__device__ __forceinline__ float sq4(const float4& v, float m) {
    const float a = v.x - m, b = v.y - m, c = v.z - m, d = v.w - m;
    return fmaf(a, a, fmaf(b, b, fmaf(c, c, d * d)));
}

// What a product is. NORM: the row is normalised (and stats are taken), code that a plain product should not have to fetch.
// ALONE: a caller's own product, whose bias may be the output of the kernel ahead: it is asked for behind the wait, with the row.
enum Kind { PLAIN, NORM, ALONE };
// NCH: 16-level chunks per lane of a row (slice). RB: rows per task; SwiGLU pairs gate row t with up row t.
template <int NCH, int RB, bool SCALED, Kind KIND>
__global__ void __launch_bounds__(MAX_WARPS * 32, 1) gemv_row_kernel(const RowArgs a) {
    extern __shared__ __align__(16) float4 xs[];             // [staged][K / 4] units of 16 bytes, swizzled
    __shared__ __align__(16) float red[3][MAX_WARPS];
    __shared__ float meet[2][MAX_WARPS][RB];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, warps = blockDim.x >> 5;
    const int K = a.K, chunks = K >> 4, units = K >> 2, kb = K >> 5;
    const int slice = wid % a.ks, per_slice = (chunks + a.ks - 1) / a.ks;
    const int c_end = min(chunks, (slice + 1) * per_slice), c0 = slice * per_slice + lane;
    const int groups = gridDim.x * (warps / a.ks);

    struct Rows { uint4 q[RB][NCH]; __half d[RB][NCH]; };
    // row of part p that slot r of task t works on; the last row again where there is none
    auto row_of = [&](int t, int r, int& p) -> int {
        if (a.epi == EPI_SWIGLU && a.parts == 2) { p = r; return t; }
        p = 0;
        while (p + 1 < a.parts) {
            const int n = (a.part[p].N + RB - 1) / RB;
            if (t < n) break;
            t -= n;
            ++p;
        }
        return t * RB + r;
    };
    auto fetch = [&](Rows& w, int t) {
        if (t >= a.tasks) return;
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            int p;
            const int n = row_of(t, r, p);
            const size_t row = (size_t)min(n, a.part[p].N - 1);
            const uint4* q = (const uint4*)(a.part[p].qu + row * K);
#pragma unroll
            for (int i = 0; i < NCH; ++i)
                if (c0 + 32 * i < c_end) {
                    w.q[r][i] = ld_levels(q + c0 + 32 * i);
                    if (SCALED) w.d[r][i] = a.part[p].d[row * kb + ((c0 + 32 * i) >> 1)];
                }
        }
    };
    Rows wa, wb;
    const int first = blockIdx.x * (warps / a.ks) + wid / a.ks;
    fetch(wa, first);

    // the first task's bias, by the lane that adds it: behind the dot product it would cost an L2 round trip
    const bool finisher = slice == 0 && lane == 0;
    float bias0[RB], res0[RB];
    auto first_bias = [&]() {
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            if (!finisher || first >= a.tasks) continue;
            int p;
            const int n = row_of(first, r, p);
            if (n < a.part[p].N && a.part[p].bias) bias0[r] = a.part[p].bias[n];
        }
    };
#pragma unroll
    for (int r = 0; r < RB; ++r) bias0[r] = res0[r] = 0.0f;
    if (KIND != ALONE) first_bias();
    // this thread's units of the norm's parameters
    const float *nw = KIND == NORM ? a.nw : nullptr, *nb = KIND == NORM ? a.nb : nullptr;
    float4 gw[UN], gb[UN];
#pragma unroll
    for (int i = 0; i < UN; ++i) {
        const int u = tid + i * blockDim.x;
        if (nw && u < units) gw[i] = ((const float4*)nw)[u];
        if (nb && u < units) gb[i] = ((const float4*)nb)[u];
    }
    // and, where the scales belong to the input index, those of its first unit (behind the wait each copy of the row would
    // cost an L2 round trip: 16 layers of width 512, int8, 64 tokens: 20.0 instead of 23.5 ms)
    float4 sx[3];
    if constexpr (!SCALED)
#pragma unroll
        for (int p = 0; p < 3; ++p)
            if (p < a.staged && a.part[p].xscale && tid < units) sx[p] = ((const float4*)a.part[p].xscale)[tid];

    pdl_wait();
    pdl_trigger();       // not ahead of the wait: what the kernel behind asks for would queue up before this one's row
    float4 v[UN];
#pragma unroll
    for (int i = 0; i < UN; ++i) {
        const int u = tid + i * blockDim.x;
        v[i] = u < units ? ((const float4*)a.x)[u] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    if (KIND == ALONE) first_bias();
    if (a.residual && finisher && first < a.tasks)
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            int p;
            const int n = row_of(first, r, p);
            if (n < a.part[p].N) res0[r] = a.residual[n];
        }
    const bool dead = a.state && (a.state->done | a.state->error);
    // stage the row: a thread's first UN units stay in registers until they are normalised, further ones are read again
    const int more = tid + UN * blockDim.x;
    float mean = 0.0f, inv = 1.0f;
    if (nw) {
        auto warp_sum = [&](float t) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            return t;
        };
        float sum = 0.0f, m_w = 0.0f, q = 0.0f;
        int n_w = 0;
        if (nb) {
            // LayerNorm: every warp takes the mean of its own elements and the squares around it; one barrier, then the warps'
            // figures are merged around the common mean (n_w (m_w - mean)^2 is what a warp's own mean left out)
#pragma unroll
            for (int i = 0; i < UN; ++i) sum += (v[i].x + v[i].y) + (v[i].z + v[i].w);
            for (int u = more; u < units; u += blockDim.x) {
                const float4 t = ((const float4*)a.x)[u];
                sum += (t.x + t.y) + (t.z + t.w);
            }
            sum = warp_sum(sum);
            for (int u = wid * 32; u < units; u += blockDim.x) n_w += 4 * min(32, units - u);
            m_w = n_w > 0 ? sum / (float)n_w : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < UN; ++i)
            if (tid + i * (int)blockDim.x < units) q += sq4(v[i], m_w);
        for (int u = more; u < units; u += blockDim.x) q += sq4(((const float4*)a.x)[u], m_w);
        q = warp_sum(q);
        if (lane == 0) { red[0][wid] = m_w; red[1][wid] = q; red[2][wid] = (float)n_w; }
        if (tid >= warps && tid < MAX_WARPS) red[0][tid] = red[1][tid] = red[2][tid] = 0.0f;
        __syncthreads();
        // every thread merges for itself: a fixed count, so that the reads are wide and the sums are trees
        auto total = [&](auto f) {
            float t[MAX_WARPS / 4];
#pragma unroll
            for (int w = 0; w < MAX_WARPS / 4; ++w) t[w] = f(((const float4*)red[0])[w], ((const float4*)red[1])[w], ((const float4*)red[2])[w]);
            return (t[0] + t[1]) + (t[2] + t[3]);
        };
        if (nb) {
            mean = total([](const float4& m, const float4&, const float4& n) { return fmaf(n.x, m.x, n.y * m.y) + fmaf(n.z, m.z, n.w * m.w); }) / (float)K;
            auto off = [&](float m, float q, float n) { const float dm = m - mean; return fmaf(n * dm, dm, q); };
            const float m2 = total([&](const float4& m, const float4& q, const float4& n) {
                return (off(m.x, q.x, n.x) + off(m.y, q.y, n.y)) + (off(m.z, q.z, n.z) + off(m.w, q.w, n.w));
            });
            inv = sqrtf(m2 / (float)K + a.eps);            // the reference divides by the deviation
        } else {
            inv = 1.0f / sqrtf(total([](const float4&, const float4& q, const float4&) { return (q.x + q.y) + (q.z + q.w); }) / (float)K + a.eps);
        }
    }
    auto put = [&](int u, float4 t, const float4& g, const float4& b) {
        if (nb) {
            t.x = ((t.x - mean) / inv) * g.x + b.x; t.y = ((t.y - mean) / inv) * g.y + b.y;
            t.z = ((t.z - mean) / inv) * g.z + b.z; t.w = ((t.w - mean) / inv) * g.w + b.w;
        } else if (nw) {
            t.x = __fmul_rn(__fmul_rn(t.x, inv), g.x); t.y = __fmul_rn(__fmul_rn(t.y, inv), g.y);
            t.z = __fmul_rn(__fmul_rn(t.z, inv), g.z); t.w = __fmul_rn(__fmul_rn(t.w, inv), g.w);
        }
        const int at = u ^ ((u >> 3) & 3);
        if (SCALED || !a.part[0].xscale) { xs[at] = t; return; }
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            if (p >= a.staged) break;
            float4 s = sx[p];
            if (u != tid) s = ((const float4*)a.part[p].xscale)[u];
            xs[(size_t)p * units + at] = make_float4(t.x * s.x, t.y * s.y, t.z * s.z, t.w * s.w);
        }
    };
#pragma unroll
    for (int i = 0; i < UN; ++i)
        if (tid + i * (int)blockDim.x < units) put(tid + i * blockDim.x, v[i], gw[i], gb[i]);
    for (int u = more; u < units; u += blockDim.x) {
        float4 g = {}, b = {};
        if (nw) g = ((const float4*)nw)[u];
        if (nb) b = ((const float4*)nb)[u];
        put(u, ((const float4*)a.x)[u], g, b);
    }
    __syncthreads();

    float top = -INFINITY, mass = 0.0f;                      // a.stats: over the outputs of this lane
    int buf = 0;
    auto work = [&](const Rows& w, int t) {
        float acc[RB];
        int p[RB], n[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) { acc[r] = 0.0f; n[r] = row_of(t, r, p[r]); }
        const bool split_x = a.staged > 1 && a.epi == EPI_SWIGLU;      // the two rows of a task have a staged row each
#pragma unroll
        for (int i = 0; i < NCH; ++i) {
            const int c = c0 + 32 * i;
            if (c < c_end) {
                const int sw = (c >> 1) & 3;
                const ulonglong2* xp = (const ulonglong2*)xs + (a.staged > 1 ? (size_t)p[0] * units : 0) + 4 * c;
                ulonglong2 x0 = xp[0 ^ sw], x1 = xp[1 ^ sw], x2 = xp[2 ^ sw], x3 = xp[3 ^ sw];
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    if (r > 0 && split_x) { xp += units; x0 = xp[0 ^ sw]; x1 = xp[1 ^ sw]; x2 = xp[2 ^ sw]; x3 = xp[3 ^ sw]; }
                    const float v = dot16x(w.q[r][i], x0, x1, x2, x3);
                    acc[r] = SCALED ? fmaf(__half2float(w.d[r][i]), v, acc[r]) : acc[r] + v;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < RB; ++r)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
        if (a.ks > 1) {
            // the slices of a row meet in slice order
            if (lane == 0)
#pragma unroll
                for (int r = 0; r < RB; ++r) meet[buf][wid][r] = acc[r];
            asm volatile("bar.sync %0, %1;" ::"r"(1 + wid / a.ks), "r"(32 * a.ks) : "memory");
            if (slice == 0)
#pragma unroll
                for (int r = 0; r < RB; ++r)
                    for (int s = 1; s < a.ks; ++s) acc[r] += meet[buf][wid + s][r];
            buf ^= 1;
        }
        if (!finisher || dead) return;
#pragma unroll
        for (int r = 0; r < RB; ++r)
            if (t == first) acc[r] += bias0[r];
            else if (a.part[p[r]].bias && n[r] < a.part[p[r]].N) acc[r] += a.part[p[r]].bias[n[r]];
        if (RB == 2 && a.epi == EPI_SWIGLU) {
            a.part[0].out[t] = __fmul_rn(__fdiv_rn(acc[0], __fadd_rn(1.0f, expf(-acc[0]))), acc[RB - 1]);
            return;
        }
#pragma unroll
        for (int r = 0; r < RB; ++r)
            if (n[r] < a.part[p[r]].N) {
                float v = acc[r];
                if (a.epi == EPI_GELU) v = gelu_f(v);
                if (a.residual) v = (t == first ? res0[r] : a.residual[n[r]]) + v;
                a.part[p[r]].out[n[r]] = v;
                if (KIND == NORM && a.stats) {
                    if (v > top) { mass *= expf(top - v); top = v; }
                    if (v != -INFINITY) mass += expf(v - top);
                }
            }
    };
    for (int t = first; t < a.tasks; t += 2 * groups) {
        fetch(wb, t + groups);
        work(wa, t);
        if (t + groups < a.tasks) {
            fetch(wa, t + 2 * groups);
            work(wb, t + groups);
        }
    }
    if (KIND == NORM && a.stats) {
        __syncthreads();
        if (lane == 0) { red[0][wid] = top; red[1][wid] = mass; }
        __syncthreads();
        if (tid == 0) {
            for (int w = 1; w < warps; ++w) top = fmaxf(top, red[0][w]);
            mass = 0.0f;
            for (int w = 0; w < warps; ++w)
                if (red[1][w] != 0.0f) mass += red[1][w] * expf(red[0][w] - top);
            a.stats[blockIdx.x] = make_float2(top, mass);
        }
    }
}

template <int NCH, int RB, bool SCALED, Kind KIND>
int launch_row_t(const RowArgs& a, int blocks, int threads, size_t smem, int dev, cudaStream_t st) {
    static bool ready[64] = {};
    if (!ready[dev]) {
        FC_CUDA(cudaFuncSetAttribute(gemv_row_kernel<NCH, RB, SCALED, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
        ready[dev] = true;
    }
    FC_CUDA(launch_pdl(gemv_row_kernel<NCH, RB, SCALED, KIND>, dim3(blocks), dim3(threads), smem, st, a));
    ++g_launches;
    return FC_OK;
}
template <int NCH>
int launch_row(int rb, bool scaled, const RowArgs& a, int blocks, int threads, size_t smem, int dev, cudaStream_t st) {
    auto go = [&](auto f) { return f(a, blocks, threads, smem, dev, st); };
    auto of = [&](auto kind) {
        constexpr Kind KIND = decltype(kind)::value;
        if (scaled) return go(rb == 2 ? launch_row_t<NCH, 2, true, KIND> : launch_row_t<NCH, 1, true, KIND>);
        return go(rb == 2 ? launch_row_t<NCH, 2, false, KIND> : launch_row_t<NCH, 1, false, KIND>);
    };
    if (a.nw) return of(std::integral_constant<Kind, NORM>());
    // without the state of a decode step the product is a caller's own, on the caller's pointers
    if (!a.state) return of(std::integral_constant<Kind, ALONE>());
    return of(std::integral_constant<Kind, PLAIN>());
}

}  // namespace

int launch_gemv_row(const GemvPart* parts, int n_parts, int K, const float* x, const RowNorm& norm, const float* residual, int epi,
                    const StepState* state, cudaStream_t st, float2* stats, int* n_stats) {
    if (n_parts < 1 || n_parts > 3 || K % 32 || K > 12288) return fail(FC_E_SHAPE, "gemv_row: %d parts, K = %d", n_parts, K);
    static int sms[64] = {};
    int dev = 0;
    FC_CUDA(cudaGetDevice(&dev));
    if (dev >= 64) return fail(FC_E_ARG, "device index %d", dev);
    if (!sms[dev]) FC_CUDA(cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev));
    RowArgs a = {};
    long rows = 0;
    for (int p = 0; p < n_parts; ++p) { a.part[p] = parts[p]; rows += parts[p].N; }
    a.parts = n_parts; a.K = K; a.x = x; a.nw = norm.w; a.nb = norm.b; a.eps = norm.eps; a.stats = stats; a.residual = residual; a.epi = epi; a.state = state;
    a.staged = parts[0].xscale ? n_parts : 1;
    if (epi == EPI_SWIGLU && (residual || n_parts > 2 || (n_parts == 1 && (parts[0].N & 1)) || (n_parts == 2 && parts[0].N != parts[1].N)))
        return fail(FC_E_SHAPE, "the SwiGLU epilogue pairs rows and takes no residual");
    if (stats && !norm.w) return fail(FC_E_ARG, "gemv_row: stats belong to a product with a norm");
    if (residual && n_parts > 1) return fail(FC_E_SHAPE, "gemv_row: a residual belongs to a single matrix");
    a.ks = K <= SLICE ? 1 : K <= 2 * SLICE ? 2 : K <= 4 * SLICE ? 4 : 8;
    const int per_slice = (K / 16 + a.ks - 1) / a.ks, nch = (per_slice + 31) / 32;
    // two rows a task when every warp of the GPU gets at least two such tasks (they share the reads of the staged row)
    const int rb = epi == EPI_SWIGLU || rows * a.ks >= 4L * MAX_WARPS * sms[dev] ? 2 : 1;
    a.tasks = 0;
    for (int p = 0; p < n_parts; ++p) a.tasks += (parts[p].N + rb - 1) / rb;
    if (epi == EPI_SWIGLU && n_parts == 2) a.tasks = parts[0].N;
    // few tasks: few warps per CTA, on all SMs
    int warps = (int)std::min<long>(MAX_WARPS, ((long)a.tasks * a.ks + sms[dev] - 1) / sms[dev]);
    warps = std::max((int)a.ks, (std::max(warps, 4) + a.ks - 1) / a.ks * a.ks);
    const int blocks = std::min(sms[dev], (a.tasks * a.ks + warps - 1) / warps);
    if (n_stats) *n_stats = blocks;
    const size_t smem = (size_t)a.staged * K * 4;
    const bool scaled = parts[0].d != nullptr;
    auto go = nch == 1 ? launch_row<1> : nch == 2 ? launch_row<2> : nch == 3 ? launch_row<3> : launch_row<4>;
    return go(rb, scaled, a, blocks, warps * 32, smem, dev, st);
}

}  // namespace fc
