// One activation row against a matrix of many rows: the standalone M = 1 linear on a vocabulary head and the like.
//
//     y[n] = bias[n] + sum_k x[k] * w[n][k]
//
// gemv_row.cu is made for a chain: a warp per row, a CTA per SM, every weight asked for ahead of the wait. With many thousand rows that
// leaves 16 warps an SM to hide a level's conversion and product, two rows to share a read of the staged row, and lanes without a
// chunk where K is no multiple of 512. Here a half warp takes ROWS rows (the staged row is read once for all), its 16 lanes cover 256
// levels of each with DEPTH such chunks in flight, and the blocks are small and many. Bound: issue and shared-memory reads (4.2
// TB/s at 50257 x 768 out of L2). A file of its own, so that the kernels of the chain keep their image.
#include "fc_common.cuh"
#include "pdl.cuh"

namespace fc {

namespace {

constexpr int THREADS = 256, HALVES = THREADS / 16;

template <int B>
__device__ __forceinline__ float qbyte(uint32_t w) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540 + B)) - 8388736.0f;
}
__device__ __forceinline__ float dot16(const uint4& w, const float4& x0, const float4& x1, const float4& x2, const float4& x3) {
    float a = x0.x * qbyte<0>(w.x), b = x1.x * qbyte<0>(w.y), c = x2.x * qbyte<0>(w.z), e = x3.x * qbyte<0>(w.w);
    a = fmaf(x0.y, qbyte<1>(w.x), a); b = fmaf(x1.y, qbyte<1>(w.y), b); c = fmaf(x2.y, qbyte<1>(w.z), c); e = fmaf(x3.y, qbyte<1>(w.w), e);
    a = fmaf(x0.z, qbyte<2>(w.x), a); b = fmaf(x1.z, qbyte<2>(w.y), b); c = fmaf(x2.z, qbyte<2>(w.z), c); e = fmaf(x3.z, qbyte<2>(w.w), e);
    a = fmaf(x0.w, qbyte<3>(w.x), a); b = fmaf(x1.w, qbyte<3>(w.y), b); c = fmaf(x2.w, qbyte<3>(w.z), c); e = fmaf(x3.w, qbyte<3>(w.w), e);
    return (a + b) + (c + e);
}
__device__ __forceinline__ uint4 ld_levels(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// SCALED: an f16 scale per 32 levels. Without, the scale belongs to the input index and is folded into the staged row.
template <bool SCALED, int ROWS, int DEPTH>
__global__ void __launch_bounds__(THREADS) gemv_wide_kernel(const GemvPart p, int K, const float* x) {
    extern __shared__ __align__(16) float4 xs[];              // 16-byte units of the row, swizzled: 16 lanes 64 bytes apart meet no bank twice
    pdl_trigger();
    const int hl = threadIdx.x & 15, row0 = (blockIdx.x * HALVES + (threadIdx.x >> 4)) * ROWS, chunks = K >> 4, kb = K >> 5;
    const bool live = row0 < p.N;                             // rows past N up to the padding are zeros
    struct Chunk { uint4 q[ROWS]; __half d[ROWS]; };
    auto fetch = [&](Chunk& w, int c) {
        if (!live || c >= chunks) return;
#pragma unroll
        for (int r = 0; r < ROWS; ++r) {
            w.q[r] = ld_levels((const uint4*)(p.qu + (size_t)(row0 + r) * K) + c);
            if (SCALED) w.d[r] = p.d[(size_t)(row0 + r) * kb + (c >> 1)];
        }
    };
    Chunk w[DEPTH];
#pragma unroll
    for (int i = 0; i < DEPTH; ++i) fetch(w[i], hl + 16 * i);
    pdl_wait();
    for (int u = threadIdx.x; u < (K >> 2); u += THREADS) {
        float4 v = ((const float4*)x)[u];
        if (!SCALED) {
            const float4 s = ((const float4*)p.xscale)[u];
            v = make_float4(v.x * s.x, v.y * s.y, v.z * s.z, v.w * s.w);
        }
        xs[u ^ ((u >> 3) & 3)] = v;
    }
    __syncthreads();
    if (!live) return;                                        // a half warp as a whole: the shuffles stay inside it
    float acc[ROWS] = {};
    for (int c0 = hl; c0 < chunks; c0 += 16 * DEPTH)
#pragma unroll
        for (int i = 0; i < DEPTH; ++i) {
            const int c = c0 + 16 * i;
            if (c >= chunks) break;
            const int sw = (c >> 1) & 3;
            const float4 x0 = xs[4 * c + (0 ^ sw)], x1 = xs[4 * c + (1 ^ sw)], x2 = xs[4 * c + (2 ^ sw)], x3 = xs[4 * c + (3 ^ sw)];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                const float v = dot16(w[i].q[r], x0, x1, x2, x3);
                acc[r] = SCALED ? fmaf(__half2float(w[i].d[r]), v, acc[r]) : acc[r] + v;
            }
            fetch(w[i], c + 16 * DEPTH);
        }
    const unsigned half = 0xFFFFu << (threadIdx.x & 16);
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(half, acc[r], o);
    const int n = row0 + hl;
    if (hl < ROWS && n < p.N) {
        float v = acc[0];
#pragma unroll
        for (int r = 1; r < ROWS; ++r) v = hl == r ? acc[r] : v;
        p.out[n] = p.bias ? v + p.bias[n] : v;
    }
}

}  // namespace

// Us in a graph, gemv_row / two rows a half warp and four chunks in flight / four rows and two:
//     N 4096:   K 768   3.2 / 2.4 / 3.3   K 1024   3.1 / 2.4 / 3.8   K 2048   4.4 / 4.8 / 7.3
//     N 8192:   K 768   5.2 / 2.6 / 4.8   K 2048   7.5 / 5.1 / 11.0  K 3072  11.2 / 6.9 / 16.0
//     N 16384:  K 256   6.0 / 3.1 / 2.6  K 512   5.9 / 3.8 / 3.7   K 2048  12.6 / 9.8 / 11.8  K 3072  19.5 / 13.2 / 16.9
//     N 32000:  K 768  13.4 / 8.8 / 7.0   K 2048  21.9 / 17.3 / 17.4
//     N 50257:  K 768  20.2 / 13.1 / 9.9  K 2048  33.4 / 24.6 / 22.9
// So: gemv_row up to 4096 rows, where neither is ahead for every K, then many small blocks until there are enough of the larger
// ones, which read the staged row half as often. With input scales every block stages two rows: N 8192, K 2048 takes 6.9 / 8.0, N
// 32000 19.3 / 17.1 (four rows), so that only the larger blocks are worth it.
int launch_gemv_alone(const GemvPart& part, int K, const float* x, cudaStream_t st) {
    const bool four = part.N >= 24576 || (part.N >= 16384 && K <= 512);
    if (part.N <= 4096 || (part.xscale && !four)) return launch_gemv_row(&part, 1, K, x, RowNorm(), nullptr, EPI_NONE, nullptr, st);
    const dim3 grid((part.N + (four ? 4 : 2) * HALVES - 1) / ((four ? 4 : 2) * HALVES));
    auto kernel = part.xscale ? gemv_wide_kernel<false, 4, 2> : four ? gemv_wide_kernel<true, 4, 2> : gemv_wide_kernel<true, 2, 4>;
    FC_CUDA(launch_pdl(kernel, grid, dim3(THREADS), (size_t)K * 4, st, part, K, x));
    ++g_launches;
    return FC_OK;
}

}  // namespace fc
