// The standalone linears (fc_q8_0_linear_dev, fc_rowq_linear_dev) with one row against a matrix of many, or with few rows:
//
//     y[m][n] = bias[n] + sum_k x[m][k] * w[n][k]
//
// gemv_row.cu is made for a chain: a warp per row, a CTA per SM, every weight asked for ahead of the wait. With many thousand rows that
// leaves 16 warps an SM to hide a level's conversion and product, two rows to share a read of the staged row, and lanes without a
// chunk where K is no multiple of 512. Here a half warp takes ROWS rows of the matrix (the staged activations are read once for all), its
// 16 lanes cover 256 levels of each with DEPTH such chunks in flight, and the blocks are small and many. Bound: issue and
// shared-memory reads (4.2 TB/s at 50257 x 768 out of L2). With few activation rows a level is converted once for MT of them;
// the tensor-core GEMM needs 7 to 13 us for any product (planes, a cluster's start, its pipeline's fill) where this takes 2 to 5.
// A file of its own, so that the kernels of the chain keep their image.
#include "fc_common.cuh"
#include "pdl.cuh"

namespace fc {

namespace {

constexpr int THREADS = 256, HALVES = THREADS / 16;

template <int B>
__device__ __forceinline__ float qbyte(uint32_t w) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7540 + B)) - 8388736.0f;
}
// 16 levels against 16 activations.
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

// The same for rows m0 .. m0 + MT of x: a level is converted once for all of them.
template <bool SCALED, int MT>
__global__ void __launch_bounds__(THREADS) gemm_few_kernel(const GemvPart p, int K, int M, const float* x) {
    constexpr int ROWS = 2, DEPTH = 2;
    extern __shared__ __align__(16) float4 xs[];              // [MT][K / 4] units, swizzled as above
    pdl_trigger();
    const int hl = threadIdx.x & 15, row0 = (blockIdx.x * HALVES + (threadIdx.x >> 4)) * ROWS, chunks = K >> 4, kb = K >> 5, units = K >> 2;
    const int m0 = blockIdx.y * MT, mt = min(MT, M - m0);
    const bool live = row0 < p.N;
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
    const float4* x4 = (const float4*)(x + (size_t)m0 * K);
    for (int u = threadIdx.x; u < units * MT; u += THREADS) {
        const int m = u / units, v = u - m * units;
        float4 t = m < mt ? x4[u] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (!SCALED) {
            const float4 s = ((const float4*)p.xscale)[v];
            t = make_float4(t.x * s.x, t.y * s.y, t.z * s.z, t.w * s.w);
        }
        xs[m * units + (v ^ ((v >> 3) & 3))] = t;
    }
    __syncthreads();
    if (!live) return;
    float acc[MT][ROWS] = {};
    for (int c0 = hl; c0 < chunks; c0 += 16 * DEPTH)
#pragma unroll
        for (int i = 0; i < DEPTH; ++i) {
            const int c = c0 + 16 * i;
            if (c >= chunks) break;
            float f[ROWS][16], d[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                const uint32_t q[4] = {w[i].q[r].x, w[i].q[r].y, w[i].q[r].z, w[i].q[r].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    f[r][4 * j] = qbyte<0>(q[j]); f[r][4 * j + 1] = qbyte<1>(q[j]);
                    f[r][4 * j + 2] = qbyte<2>(q[j]); f[r][4 * j + 3] = qbyte<3>(q[j]);
                }
                d[r] = SCALED ? __half2float(w[i].d[r]) : 1.0f;
            }
            fetch(w[i], c + 16 * DEPTH);
            const int sw = (c >> 1) & 3;
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float4* xp = xs + m * units + 4 * c;
                float s[ROWS][2] = {};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 v = xp[j ^ sw];
#pragma unroll
                    for (int r = 0; r < ROWS; ++r) {
                        float& t = s[r][j & 1];
                        t = fmaf(v.x, f[r][4 * j], t); t = fmaf(v.y, f[r][4 * j + 1], t);
                        t = fmaf(v.z, f[r][4 * j + 2], t); t = fmaf(v.w, f[r][4 * j + 3], t);
                    }
                }
#pragma unroll
                for (int r = 0; r < ROWS; ++r) acc[m][r] = fmaf(d[r], s[r][0] + s[r][1], acc[m][r]);
            }
        }
    const unsigned half = 0xFFFFu << (threadIdx.x & 16);
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int r = 0; r < ROWS; ++r)
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) acc[m][r] += __shfl_xor_sync(half, acc[m][r], o);
    float v = acc[0][0];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int r = 0; r < ROWS; ++r) v = hl == m * ROWS + r ? acc[m][r] : v;
    const int m = hl / ROWS, n = row0 + hl % ROWS;
    if (m < mt && n < p.N) p.out[(size_t)(m0 + m) * p.N + n] = p.bias ? v + p.bias[n] : v;
}

constexpr int FEW = 4, FEW_K = 48 * 1024 / 4 / FEW;           // activation rows of a block, and the K at which they fill its memory

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


// Whether M >= 2 rows are better off here than on the tensor-core GEMM. Us in a graph, GEMM / here:
//     M 4:   N 500, K 96   7.4 / 2.0   N 2304, K 768  14.7 / 3.8   N 4096, K 1024  9.9 / 5.0   N 16384, K 2048  26.5 / 17.6
//     M 8:   N 500, K 96   7.5 / 2.1   N 2304, K 768  14.8 / 4.5   N 4096, K 1024  9.9 / 5.3   N 16384, K 2048  26.5 / 31.6
//     M 16:  N 768, K 768  8.9 / 4.2   N 768, K 3072  11.5 / 11.4  N 4096, K 1024 10.0 / 9.9   N 4096, K 128     8.0 / 4.5
//     M 32:  N 768, K 768  8.9 / 4.7   N 768, K 3072  11.5 / 12.5  N 4096, K 1024 10.6 / 16.8  N 4096, K 128     8.1 / 8.2
// So up to four rows always, more while they take fewer than 2^25 products (a half warp passes over 256 of k at a time).
bool few_rows(int N, int K, int M) {
    return K <= FEW_K && (M <= FEW || (double)M * N * ((K + 255) / 256 * 256) < (double)(1 << 25));
}

// M rows of a caller's own product without scratch: few of them, or any number where there is no memory for the planes.
int launch_rows_alone(GemvPart part, int K, const float* x, int M, cudaStream_t st) {
    const int step = K <= FEW_K ? 65535 * FEW : 1;
    for (int m0 = 0; m0 < M; m0 += step, x += (size_t)step * K, part.out += (size_t)step * part.N) {
        if (M == 1 || step == 1) {
            FC_TRY(launch_gemv_alone(part, K, x, st));
            continue;
        }
        const int m = M - m0 < step ? M - m0 : step, mt = m == 2 ? 2 : FEW;
        const dim3 grid((part.N + 2 * HALVES - 1) / (2 * HALVES), (m + mt - 1) / mt);
        auto kernel = part.xscale ? (mt == 2 ? gemm_few_kernel<false, 2> : gemm_few_kernel<false, FEW>)
                                  : (mt == 2 ? gemm_few_kernel<true, 2> : gemm_few_kernel<true, FEW>);
        FC_CUDA(launch_pdl(kernel, grid, dim3(THREADS), (size_t)mt * K * 4, st, part, K, m, x));
        ++g_launches;
    }
    return FC_OK;
}

}  // namespace fc
