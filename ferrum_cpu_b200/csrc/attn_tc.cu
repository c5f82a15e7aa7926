// Causal multi-head attention of a full window on the tcgen05 tensor cores (head_dim 64).
//
// Replaces the per-(window, head) loop of TransformerBlock::forward
// (ferrum_core/src/layer/transformer.rs:395-477): S = Q Kᵀ / sqrt(hd), entries j > i masked,
// row softmax, O = P V. The T x T probability matrix the reference keeps (`last_attention`,
// transformer.rs:458-478) is never formed: keys are visited in tiles of 64 with an online
// softmax. Both products run on bf16 planes with fp32 accumulation: with two planes as three products (q1·k1 + q1·k2 +
// q2·k1; the same for P·V, so they reproduce f32 products to 2^-16 relative), with three planes (the f32 math mode) as six
// (all of order up to 2^-16; what is dropped is 2^-24 of a product). Two f16 planes of a scale times the values (gemm_f16.cu) take the
// same three products as two of bf16 and hold 2^-23.
//
// Inputs are the bf16 planes of the fused qkv rows [R][3d] written by the QKV GEMM; the output are the planes [R][d] the
// out-projection GEMM reads. Windows of a batch may differ in length: they lie one after the other without padding.
//
// One CTA owns 128 query rows of one (window, head); with two planes two CTAs fit on an SM, so one's softmax overlaps the
// other's MMAs.
//   warps 0-3   one query row per thread: tcgen05.ld the score tile, scale, mask, running
//               max / sum, write P (bf16 planes, 128-byte swizzle) to shared memory, then
//               fold the P·V tile into the row's output registers;
//   warp 4      TMA: Q once, then a K tile and a V tile (64 keys) per step;
//   warp 5      tcgen05.mma issue: 12 (24) MMAs for the score tile, as many for P·V (V is consumed
//               MN-major, exactly as TMA lays out its [keys][hd] rows).
// Every mbarrier wait is bounded; on a timeout the status word is raised and the CTA leaves, each warp as a whole.
//
// Bound: tensor pipe / MUFU. 4·hd·T(T+1)/2 algorithmic FLOP per (window, head).
#include "pdl.cuh"
#include "tc.cuh"

namespace fc {

namespace {

constexpr int HD = 64;                 // head dimension
constexpr int QT = 128;                // query rows per CTA
constexpr int KT = 64;                 // keys per step
constexpr int Q_BYTES = QT * HD * 2;   // one bf16 plane of the Q tile: 16 KiB
constexpr int KV_BYTES = KT * HD * 2;  // one bf16 plane of a K or V tile: 8 KiB
constexpr int P_BYTES = QT * KT * 2;   // one bf16 plane of the P tile: 16 KiB
// Shared memory of a CTA that works on P planes: 96 KB for two (two CTAs per SM), 144 KB for three.
template <int P>
struct Smem {
    static constexpr int Q = 0, K = Q + P * Q_BYTES, V = K + P * KV_BYTES, PR = V + P * KV_BYTES, BARS = PR + P * P_BYTES;
};
constexpr int SOFTMAX_WARPS = 4, TMA_WARP = 4, MMA_WARP = 5, THREADS = 6 * 32;
constexpr int TMEM_COLS = 128;         // score tile: columns 0..63, P·V tile: columns 64..127
// f32 sums, M = 128, N = 64; B K-major for Q·Kᵀ, MN-major (bit 16) for P·V
constexpr uint32_t BF16 = (1u << 7) | (1u << 10);        // operand types; without: f16
constexpr uint32_t IDESC_S = (1u << 4) | ((uint32_t)(KT >> 3) << 17) | ((uint32_t)(QT >> 4) << 24);
constexpr uint32_t IDESC_O = (1u << 4) | (1u << 16) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(QT >> 4) << 24);

struct Bars {
    unsigned long long q_full, k_full, v_full, k_empty, v_empty;
    unsigned long long s_full, s_empty, p_full, o_full, o_empty;
    uint32_t tmem_base;
    volatile int abort;
};
template <int P>
constexpr int SMEM_BYTES = Smem<P>::BARS + 1024 /* alignment slack */ + (int)sizeof(Bars);

__device__ __forceinline__ uint32_t s32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 2^x on the special-function unit (2 ulp); 2^-inf = 0
__device__ __forceinline__ float ex2_approx(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ void mbar_init(unsigned long long* b, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(s32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned long long* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(s32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s32(b)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned long long* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(s32(b)), "r"(parity), "r"(2000u) : "memory");
    return ok != 0;
}
template <class Args>
__device__ bool wait_bar(Bars* bars, unsigned long long* b, uint32_t parity, const Args& a) {
    const long long t0 = clock64();
    while (!mbar_try_wait(b, parity)) {
        if (bars->abort) return false;
        if (clock64() - t0 > a.wait_cycles) {
            tc::give_up(&bars->abort, a);
            return false;
        }
    }
    return true;
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, unsigned long long* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(s32(dst)), "l"(map), "r"(x), "r"(y), "r"(s32(bar)) : "memory");
}
// 128-byte swizzle, 8-row atoms of 1024 bytes (SBO = 64 x 16 B), descriptor version 1. The same
// encoding serves K-major tiles (rows = M or N index) and the MN-major V tile (rows = keys).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)64 << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(s32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// The products of planes i and j that a P-plane product keeps (i + j < P), the smallest first: they meet a small accumulator.
template <int P, class F>
__device__ __forceinline__ void each_term(F f) {
#pragma unroll
    for (int order = P - 1; order >= 0; --order)
#pragma unroll
        for (int i = 0; i <= order; ++i) f(i, order - i, order == P - 1 && i == 0);
}

struct AttnArgs {
    Windows win;
    int k_col, v_col;            // first column of the key / value heads in the fused q | k | v planes
    int group;                   // query heads per key / value head (1: multi-head attention)
    int ldo;                     // row stride of the output planes (= query heads x 64)
    uint16_t* out[3];            // [R][ldo] bf16 planes, or
    float unscale;               // f16 planes: 1 / their scale
    float out_scale, out_lo;     // not 0: f16 planes of out_scale times the output, the second times out_lo
    int* status;
    long long wait_cycles;       // budget of every mbarrier wait
    int withhold;                // test hook: 1: nothing is copied
};

}  // namespace

struct AttnMaps { CUtensorMap q[3], kv[3]; };    // per plane: boxes of 128 query rows, of 64 key rows

// F16: two f16 planes of a scale times the values, else bf16 planes.
template <int P, bool F16>
__global__ void __launch_bounds__(THREADS, P == 2 ? 2 : 1)
attn_prefill_tc_kernel(const __grid_constant__ AttnMaps maps, const AttnArgs a) {
    constexpr int OFF_Q = Smem<P>::Q, OFF_K = Smem<P>::K, OFF_V = Smem<P>::V, OFF_P = Smem<P>::PR, OFF_BARS = Smem<P>::BARS;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    Bars* bars = (Bars*)(smem + OFF_BARS);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int qt = (gridDim.x - 1) - blockIdx.x;          // long (late) query tiles first
    const int h = blockIdx.y, b = blockIdx.z;
    const int T = a.win.length(b), row0 = a.win.begin(b); // the window's rows in [R]
    const int q0 = qt * QT;                               // first query of the tile inside the window
    if (q0 >= T) {                                        // a window shorter than the longest
        pdl_wait();
        return;
    }
    const int last_q = min(T, q0 + QT) - 1;               // last valid query
    const int n_kt = last_q / KT + 1;                     // key tiles 0..n_kt-1 cover keys 0..last_q

    if (threadIdx.x == 0) {
        mbar_init(&bars->q_full, 1);
        mbar_init(&bars->k_full, 1); mbar_init(&bars->v_full, 1);
        mbar_init(&bars->k_empty, 1); mbar_init(&bars->v_empty, 1);
        mbar_init(&bars->s_full, 1); mbar_init(&bars->s_empty, SOFTMAX_WARPS);
        mbar_init(&bars->p_full, SOFTMAX_WARPS);
        mbar_init(&bars->o_full, 1); mbar_init(&bars->o_empty, SOFTMAX_WARPS);
        bars->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(&bars->tmem_base)), "r"((uint32_t)TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, bars->tmem_base, 0);
    pdl_wait();                                           // set up while the kernel ahead still ran
    pdl_trigger();

    if (warp == TMA_WARP) {
        if (a.withhold != 1 && tc::elect_one()) {
            mbar_expect_tx(&bars->q_full, P * Q_BYTES);
#pragma unroll
            for (int p = 0; p < P; ++p) tma_load_2d(smem + OFF_Q + p * Q_BYTES, &maps.q[p], h * HD, row0 + q0, &bars->q_full);
            for (int kt = 0; kt < n_kt; ++kt) {
                const uint32_t par = (kt & 1) ^ 1;
                if (!wait_bar(bars, &bars->k_empty, par, a)) break;
                mbar_expect_tx(&bars->k_full, P * KV_BYTES);
#pragma unroll
                for (int p = 0; p < P; ++p) tma_load_2d(smem + OFF_K + p * KV_BYTES, &maps.kv[p], a.k_col + (h / a.group) * HD, row0 + kt * KT, &bars->k_full);
                if (!wait_bar(bars, &bars->v_empty, par, a)) break;
                mbar_expect_tx(&bars->v_full, P * KV_BYTES);
#pragma unroll
                for (int p = 0; p < P; ++p) tma_load_2d(smem + OFF_V + p * KV_BYTES, &maps.kv[p], a.v_col + (h / a.group) * HD, row0 + kt * KT, &bars->v_full);
            }
        }
    } else if (warp == MMA_WARP) {
        if (tc::elect_one()) {
            const uint32_t sb = s32(smem);
            const uint64_t dq = smem_desc(sb + OFF_Q), dk = smem_desc(sb + OFF_K), dv = smem_desc(sb + OFF_V), dp = smem_desc(sb + OFF_P);
            constexpr uint64_t QS = Q_BYTES / 16, KS = KV_BYTES / 16, PS = P_BYTES / 16;   // from plane to plane, in descriptor units
            bool ok = wait_bar(bars, &bars->q_full, 0, a);
            // score tile kt: its keys have landed and the softmax warps have read the previous one out of TMEM
            auto issue_scores = [&](int kt) -> bool {
                const uint32_t par = kt & 1;
                if (!(wait_bar(bars, &bars->k_full, par, a) && wait_bar(bars, &bars->s_empty, par ^ 1, a))) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                each_term<P>([&](int i, int j, bool first) {
#pragma unroll
                    for (int ks = 0; ks < HD / 16; ++ks)                        // 32 bytes along hd per step
                        umma(tmem, dq + i * QS + ks * 2, dk + j * KS + ks * 2, IDESC_S | (F16 ? 0u : BF16), !(first && ks == 0));
                });
                umma_commit(&bars->s_full);
                umma_commit(&bars->k_empty);
                return true;
            };
            ok = ok && issue_scores(0);
            for (int kt = 0; kt < n_kt && ok; ++kt) {
                const uint32_t par = kt & 1;
                // the next score tile is issued ahead of this tile's P·V: its MMAs run while the softmax warps are
                // still turning this tile's scores into P, and its scores are ready when they come back
                if (kt + 1 < n_kt) {
                    ok = issue_scores(kt + 1);
                    if (!ok) break;
                }
                // P·V tile: P is in shared memory, the previous P·V tile has been folded in
                ok = wait_bar(bars, &bars->v_full, par, a) && wait_bar(bars, &bars->p_full, par, a) &&
                     wait_bar(bars, &bars->o_empty, par ^ 1, a);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                each_term<P>([&](int i, int j, bool first) {
#pragma unroll
                    for (int ks = 0; ks < KT / 16; ++ks)                        // 32 bytes along the keys of a P row, 16 key rows of 128 bytes of V
                        umma(tmem + HD, dp + i * PS + ks * 2, dv + j * KS + ks * 128, IDESC_O | (F16 ? 0u : BF16), !(first && ks == 0));
                });
                umma_commit(&bars->o_full);
                umma_commit(&bars->v_empty);
            }
        }
    } else {
        // ------------------------------------------------------------------ softmax warps
        const int r = warp * 32 + lane;               // query row inside the tile
        const int qi = q0 + r;                        // query index inside the window
        const float c2 = 0.125f * 1.4426950408889634f * (F16 ? a.unscale * a.unscale : 1.0f);   // 1 / sqrt(64) times log2(e)
        // f16 planes of 2^12 times the probabilities (the mass with them), so that the second plane of a small one is not lost
        constexpr float LIFT = F16 ? 12.0f : 0.0f;
        float o[HD];
#pragma unroll
        for (int c = 0; c < HD; ++c) o[c] = 0.0f;
        float m = -INFINITY, l = 0.0f;
        unsigned char* prow = smem + OFF_P + r * 128;
        const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);
        bool ok = true;
        for (int kt = 0; kt < n_kt && ok; ++kt) {
            const uint32_t par = kt & 1;
            ok = __all_sync(0xffffffffu, wait_bar(bars, &bars->s_full, par, a));   // loads, votes and barriers below are a warp's
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t s0[32], s1[32];
            tmem_ld32(lane_addr, s0);
            tmem_ld32(lane_addr + 32, s1);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->s_empty);
            // causal mask (key j > query i has weight exactly 0) and running max on the raw scores; the scale
            // 1 / sqrt(hd) and log2(e) go into one constant of the exponent: p = 2^((s - max) * scale * log2 e)
            const int k0 = kt * KT;
            float sv[KT];
            float tmax = -INFINITY;
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                sv[j] = (k0 + j <= qi) ? __uint_as_float(s0[j]) : -INFINITY;
                sv[32 + j] = (k0 + 32 + j <= qi) ? __uint_as_float(s1[j]) : -INFINITY;
                tmax = fmaxf(tmax, fmaxf(sv[j], sv[32 + j]));
            }
            const float mn = fmaxf(m, tmax);          // finite from the first tile on (key 0 <= every query)
            const float corr = exp2f((m - mn) * c2);
            const float off2 = LIFT - mn * c2;
            float psum = 0.0f;
#pragma unroll
            for (int c = 0; c < KT / 8; ++c) {        // 16-byte chunk c of the P row: 8 keys
                float p[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) { p[e] = ex2_approx(fmaf(sv[8 * c + e], c2, off2)); psum += p[e]; }
                uint32_t w[4][P];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if constexpr (F16) split2_f16(p[2 * e], p[2 * e + 1], 1.0f, w[e]);
                    else split2<P>(p[2 * e], p[2 * e + 1], w[e]);
                }
#pragma unroll
                for (int t = 0; t < P; ++t)        // 128-byte swizzle
                    *(uint4*)(prow + t * P_BYTES + (c ^ (r & 7)) * 16) = make_uint4(w[0][t], w[1][t], w[2][t], w[3][t]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->p_full);
            l = fmaf(l, corr, psum);
            m = mn;
            if (__any_sync(0xffffffffu, corr != 1.0f)) {   // the running max moves in the first tiles and rarely after
#pragma unroll
                for (int c = 0; c < HD; ++c) o[c] *= corr;
            }
            // fold in this tile's P·V
            ok = __all_sync(0xffffffffu, wait_bar(bars, &bars->o_full, par, a));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            tmem_ld32(lane_addr + HD, s0);
            tmem_ld32(lane_addr + HD + 32, s1);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->o_empty);
#pragma unroll
            for (int c = 0; c < 32; ++c) { o[c] += __uint_as_float(s0[c]); o[32 + c] += __uint_as_float(s1[c]); }
        }
        if (ok && qi < T) {
            const float inv = F16 ? a.unscale / l : 1.0f / l;
            const size_t off = (size_t)(row0 + qi) * a.ldo + (size_t)h * HD;
#pragma unroll
            for (int c = 0; c < HD / 8; ++c) {
                uint32_t w[4][P];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float v0 = o[8 * c + 2 * e] * inv, v1 = o[8 * c + 2 * e + 1] * inv;
                    if (a.out_scale != 0.0f) {
                        uint32_t t[2];
                        split2_f16(v0 * a.out_scale, v1 * a.out_scale, a.out_lo, t);
                        w[e][0] = t[0]; w[e][1] = t[1];
                    } else {
                        split2<P>(v0, v1, w[e]);
                    }
                }
#pragma unroll
                for (int t = 0; t < P; ++t)
                    if (a.out[t]) *(uint4*)(a.out[t] + off + 8 * c) = make_uint4(w[0][t], w[1][t], w[2][t], w[3][t]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (bars->abort) {                                     // copies and MMAs may be in flight for a few microseconds more
        const long long t0 = clock64();
        while (clock64() - t0 < 200000) __nanosleep(200);
    }
    __syncthreads();
    if (warp == MMA_WARP) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TMEM_COLS) : "memory");
    }
}

namespace {
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// A [rows][cols] bf16 plane viewed through boxes of 64 columns x box_rows rows, 128-byte swizzle.
int encode(CUtensorMap* map, const void* plane, size_t rows, size_t cols, int box_rows, bool f16) {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        FC_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
        if (!p || q != cudaDriverEntryPointSuccess) return fail(FC_E_CUDA, "cuTensorMapEncodeTiled is not available");
        fn = (EncodeTiledFn)p;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)plane, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(FC_E_CUDA, "cuTensorMapEncodeTiled failed (%d) for a [%zu][%zu] bf16 plane", (int)r, rows, cols);
    return FC_OK;
}
}  // namespace

// qkv: bf16 planes [R][H*64 + 2*KV*64] (q heads | k heads | v heads per row); out: planes [R][H*64]. Query head h reads key /
// value head h / (H / KV).
template <int P, bool F16>
static int launch_attn_tc(const Planes& qkv, const Windows& w, int R, int H, int KV, const Planes& out, int* status, cudaStream_t st) {
    if (KV <= 0 || H % KV) return fail(FC_E_DIM, "n_heads %d must be a multiple of n_kv_heads %d", H, KV);
    static bool attr_set[64] = {};
    int dev = 0;
    FC_CUDA(cudaGetDevice(&dev));
    if (dev < 64 && !attr_set[dev]) {
        FC_CUDA(cudaFuncSetAttribute(attn_prefill_tc_kernel<P, F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES<P>));
        attr_set[dev] = true;
    }
    const size_t ld = (size_t)(H + 2 * KV) * HD;
    AttnMaps maps;
    AttnArgs a;
    for (int p = 0; p < P; ++p) {
        FC_TRY(encode(&maps.q[p], qkv.p[p], R, ld, QT, F16));
        FC_TRY(encode(&maps.kv[p], qkv.p[p], R, ld, KT, F16));
        a.out[p] = p < out.n ? (uint16_t*)out.p[p] : nullptr;
    }
    a.win = w; a.k_col = H * HD; a.v_col = (H + KV) * HD; a.group = H / KV; a.ldo = H * HD;
    a.unscale = F16 ? 1.0f / qkv.scale : 1.0f;
    a.out_scale = out.scale; a.out_lo = out.lo;
    a.status = status; a.wait_cycles = g_debug.wait_cycles; a.withhold = g_debug.withhold;
    dim3 grid((w.T + QT - 1) / QT, H, w.B);
    FC_CUDA(launch_pdl(attn_prefill_tc_kernel<P, F16>, grid, dim3(THREADS), SMEM_BYTES<P>, st, maps, a));
    FC_LAUNCHED();
    return FC_OK;
}

int launch_attn_prefill_tc_gqa(const Planes& qkv, const Windows& w, int R, int H, int KV, const Planes& out, int* status, cudaStream_t st) {
    if (qkv.scale != 0.0f && qkv.lo != 1.0f) return fail(FC_E_ARG, "the attention's planes add up as they are");
    if (qkv.scale != 0.0f) return launch_attn_tc<2, true>(qkv, w, R, H, KV, out, status, st);
    return qkv.n == 3 ? launch_attn_tc<3, false>(qkv, w, R, H, KV, out, status, st) : launch_attn_tc<2, false>(qkv, w, R, H, KV, out, status, st);
}

// The multi-head form: planes [R][3d] in, [R][d] out.
int launch_attn_prefill_tc(const Planes& qkv, const Windows& w, int R, int d, int H, const Planes& out, int* status, cudaStream_t st) {
    if (d != H * HD) return fail(FC_E_SHAPE, "tensor-core attention needs head_dim 64 (d = %d, H = %d)", d, H);
    return launch_attn_prefill_tc_gqa(qkv, w, R, H, H, out, status, st);
}

}  // namespace fc
