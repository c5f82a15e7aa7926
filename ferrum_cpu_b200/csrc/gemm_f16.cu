// Q8_0 GEMM with the weight as two f16 planes:
//     Y[M][N] = X[M][K] · dequant(W[N][K])ᵀ + bias (+GELU) (+residual), or the softmax records of the LM head
//
// The product of the two-plane math mode (FC_MATH_BF16X3). A Q8_0 weight d·q has at most 19
// significant bits (11 of the f16 scale, 8 of the level) and is a whole multiple of 2^-24, so hi = f16(d·q) and lo = d·q - hi hold it
// EXACTLY, as long as d·128 does not overflow f16 (QMat::f16_exact, checked at upload). An activation, scaled by a power of two
// that keeps it in range, is hi + lo to 2^-23 relative. Three MMAs per step, hi·hi + hi·lo + lo·hi, drop 2^-24 of a product, and no
// scale is left to apply: k-blocks add up in TMEM, and the tensor pipe is what bounds the kernel. The lo planes hold kRest = 2^11 times
// their values: an element 2^28 below the largest of its row (of the scale's bound, in a window forward) still keeps 2^-23 of itself.
//
// gemm_tc.cu multiplies the levels instead (two MMAs per step with bf16 planes of x) and has to fold every 32-wide k-block
// into registers by the block's scale: its drain is what bounds it, at half the rate of the pipe, and its two bf16 planes of x
// leave 2^-17. It stays for the f32 mode (three bf16 planes are an f32 exactly, two of f16 are not: its three products here took 16 %
// off a batch of mixed requests, with a product at K = 768 at 1.08e-7 from 64 bits for 1.03e-7), for matrices that f16 does not hold, and for few
// rows of a prime or of a caller's own, which it splits over K.
//
// The tensor core truncates its f32 sums: towards zero, once per MMA, by up to an ulp of the whole sum however small what is added. So
// the small terms (hi·lo, lo·hi) have sums of their own, which 1 / kRest brings to where truncation does not count, and the sums of hi·hi
// stay in TMEM for FIRST = 6 stages of a tile, then for KGROUP = 3 at a time, and go into f32 registers, rounded to nearest. Sums that need no rounding
// lose nothing. Error against 64 bits on normal draws (relative, 2-norm) at K = 512 / 768 / 1024 / 3072 / 4096: 4.4e-7 / 4.0e-7 / 3.7e-7 / 3.2e-7 /
// 3.1e-7. Levels and two bf16 planes: 2.5e-6. All three terms in one sum, four stages: 8e-7, in groups of one stage 1.4e-7 and a tenth slower.
//
// With a place each, the 512 columns hold no second buffer. The order of a tile's MMAs makes up for it: at a group's end the drain
// reads the sums of hi·hi (some 1000 cycles from commit to issuer) while the small terms of that stage and the next group's first run, and a
// tile's first and last small terms come behind the main terms of two stages. The first group is long because the drain is in the epilogue of the
// tile before: with 4 + 4 stages 4096 x 1024 x 4096 took 102 us, 98 now (two buffers, one sum: 97).
//
// One CTA per SM, 640 threads (registers 104 a thread of the drain, 64 of the others):
//   warps 0-15  drain: a group's sums from TMEM into registers (lane = weight row, column = activation row); after the last
//               group bias / GELU / residual or the softmax records, and the stores. With 8 warps of twice the columns the GELU
//               epilogue was latency-bound: 32768 x 768 x 3072 390 us, now 298
//   warp 16     TMA: both planes of the weight and of the activations, 64 k a stage
//   warp 17     MMA issue and the TMEM allocation: up to 256 columns for the sums of hi·hi, as many for the small terms'.
//               One elected thread (tc.cuh: elect_one) issues an MMA in about 30 cycles; behind lane == 0 it took 74
// CG = 2: a pair of CTAs shares a tile of 256 weight rows (each holds 128 of them and half of the activation rows). CG = 1
// takes few rows. The order of a row's sums depends on K alone, so a row's result does not depend on the rows beside it.
//
// Bound: the tensor pipe at the clock the power limit leaves. A stage of a 256-row tile takes 1547 cycles, its MMAs 1536. In a loop of
// their own, with the planes made (levels in gemm_tc.cu): 4096 x 1024 x 4096 72 us (109), 32768 x 768 x 2304 234 us = 1.49 PFLOP/s executed
// (348), 16384 x 3072 x 768 161 us.
//
// Every wait is bounded; a wait that runs out raises the status word and all roles leave, in whatever order they learn of it.
#include <algorithm>
#include <type_traits>

#include "pdl.cuh"
#include "tc.cuh"

namespace fc {

using namespace tc;

namespace {

constexpr int BK = 64;                                  // k per stage: one 128-byte swizzle row of f16
constexpr int FIRST = 6, KGROUP = 3;                    // stages whose sums stay in TMEM: a tile's first ones, then so many at a time
static_assert(FIRST >= 2, "the first two stages of a tile are one group");
constexpr int W_BYTES = 128 * BK * 2;                   // one plane of the CTA's weight tile of a stage
constexpr int DRAIN_WARPS = 16, TMA_WARP = 16, MMA_WARP = 17, THREADS = 640;
constexpr int MAX_STAGES = 6;
constexpr int TMEM_COLS = 512, REST = 256;              // the sums of hi·hi, and from column REST on those of the small terms
constexpr int SMEM_LIMIT = 227 * 1024;

enum Mode : int { OUT_F32 = 0, OUT_PLANES = 1 /* bf16 planes, or f16 planes of a scale */, OUT_GELU = 2 /* f16 planes, after GELU */, OUT_SCORE = 3 };

struct F16Args {
    int N, K, M, stages;
    const float* bias; const float* residual; int gelu;
    float inv;                // what takes the scale of x out of a sum (a power of two)
    const float* row_inv;     // the same per activation row, or null
    float* y; int ldy;        // OUT_F32
    uint16_t* yp[3];          // OUT_PLANES, OUT_GELU: planes (three only of bf16), ldy elements apart
    float out_scale, out_lo;  // f16 planes: of out_scale times the output, the second times out_lo
    const int* targets; float4* stats; float* tlogit;      // OUT_SCORE
    int* status;
    long long wait_cycles;
    int withhold;             // test hooks
};

constexpr int BAR_FULL = 0, BAR_EMPTY = BAR_FULL + 8 * MAX_STAGES, BAR_ACC_FULL = BAR_EMPTY + 8 * MAX_STAGES, BAR_ACC_EMPTY = BAR_ACC_FULL + 8;
constexpr int BAR_REST_FULL = BAR_ACC_EMPTY + 8, BAR_REST_EMPTY = BAR_REST_FULL + 8, BAR_TMEM = BAR_REST_EMPTY + 8, BAR_ABORT = BAR_TMEM + 4, BAR_BYTES = BAR_ABORT + 4;

__device__ __forceinline__ void add2(uint64_t& acc, uint64_t v) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(v)); }

}  // namespace

// CW: columns (activation rows) of a drain warp, a quarter of the tile's.
template <int CG, int CW, int MODE>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f16_kernel(const __grid_constant__ CUtensorMap wh, const __grid_constant__ CUtensorMap wl, const __grid_constant__ CUtensorMap xh,
                const __grid_constant__ CUtensorMap xl, const F16Args a) {
    constexpr int NT = 4 * CW, XR = NT / CG;                                        // activation rows of a tile, of this CTA's memory
    constexpr int X_BYTES = XR * BK * 2, STAGE = 2 * W_BYTES + 2 * X_BYTES;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = smem_raw + ((1024 - (s32(smem_raw) & 1023)) & 1023);
    float4* recs = (float4*)(smem + a.stages * STAGE);                              // OUT_SCORE: [4 quarters][NT]
    unsigned char* tail = (unsigned char*)recs + (MODE == OUT_SCORE ? 4 * NT * 16 : 0);
    volatile int* abort = (volatile int*)(tail + BAR_ABORT);
    const uint32_t sb = s32(smem), full = s32(tail) + BAR_FULL, empty = s32(tail) + BAR_EMPTY;
    const uint32_t acc_full = s32(tail) + BAR_ACC_FULL, acc_empty = s32(tail) + BAR_ACC_EMPTY;
    const uint32_t rest_full = s32(tail) + BAR_REST_FULL, rest_empty = s32(tail) + BAR_REST_EMPTY;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int rank = CG == 2 ? (int)(blockIdx.x & 1) : 0;
    const int group = blockIdx.x / CG, n_groups = gridDim.x / CG;                   // CTAs or pairs take tiles in turn
    const int tiles_n = (a.N + 128 * CG - 1) / (128 * CG), tiles_m = (a.M + NT - 1) / NT;
    const int n_tiles = tiles_n * tiles_m;
    const int nst = (a.K + BK - 1) / BK;
    const bool leader = rank == 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(full + 8 * s, 1);
            mbar_init(empty + 8 * s, 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, DRAIN_WARPS * CG);
        mbar_init(rest_full, 1);
        mbar_init(rest_empty, DRAIN_WARPS * CG);
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tail + BAR_TMEM)), "r"((uint32_t)TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tail + BAR_TMEM)), "r"((uint32_t)TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (CG == 2) {
        __syncwarp();
        cluster_sync();
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, *(volatile uint32_t*)(tail + BAR_TMEM), 0);
    pdl_wait();                                                                     // set up while the kernel ahead still ran
    pdl_trigger();
    // the barriers the pair's MMA issuer waits on are the leader's
    const uint32_t full_leader = CG == 2 ? mapa(full, 0) : full, acc_empty_leader = CG == 2 ? mapa(acc_empty, 0) : acc_empty,
                   rest_empty_leader = CG == 2 ? mapa(rest_empty, 0) : rest_empty;

    // Every role ends here: nobody leaves while a peer may still reach this CTA's shared memory or barriers. After an
    // aborted wait, copies and MMAs may be in flight for a few microseconds more: outstay them.
    auto leave = [&]() {
        __syncwarp();
        if (*abort) {
            const long long t0 = clock64();
            while (clock64() - t0 < 200000) __nanosleep(200);
        }
        __syncwarp();
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (CG == 2) cluster_sync();
        else asm volatile("bar.sync 0, %0;" ::"n"(THREADS) : "memory");
    };

    if (warp >= TMA_WARP) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        if (warp == TMA_WARP && a.withhold != 1 && elect_one()) {
            // ------------------------------------------------------------ TMA producer
            int s = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int tile = group; tile < n_tiles && ok; tile += n_groups) {
                const int n0 = (tile % tiles_n) * (128 * CG) + rank * 128, m0 = (tile / tiles_n) * NT + rank * XR;
                for (int kb = 0; kb < nst; ++kb) {
                    ok = wait_bar(empty + 8 * s, ph, abort, a);
                    if (!ok) break;
                    const uint32_t dst = sb + s * STAGE, bar = full_leader + 8 * s;
                    if (leader) mbar_expect_tx(full + 8 * s, (uint32_t)(CG * STAGE));
                    tma_load_2d<CG>(dst, &wh, kb * BK, n0, bar);
                    tma_load_2d<CG>(dst + W_BYTES, &wl, kb * BK, n0, bar);
                    tma_load_2d<CG>(dst + 2 * W_BYTES, &xh, kb * BK, m0, bar);
                    tma_load_2d<CG>(dst + 2 * W_BYTES + X_BYTES, &xl, kb * BK, m0, bar);
                    if (++s == a.stages) { s = 0; ph ^= 1; }
                }
            }
        } else if (warp == MMA_WARP && leader && elect_one()) {
            // ------------------------------------------------------------ MMA issuer
            // f16 x f16 -> f32, M = 128 (256 for the pair), N = NT, both operands K-major
            constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(8 * CG) << 24);
            const uint64_t desc = smem_desc(sb);
            const uint32_t dhi = (uint32_t)(desc >> 32);
            const uint32_t rest = tmem + REST;
            uint32_t w = (uint32_t)desc, ph = 0, aph = 1, rph = 1;
            auto main_terms = [&](auto accumulate) {
                const uint32_t x = w + 2 * W_BYTES / 16;                            // descriptors count 16 bytes
                umma<CG, decltype(accumulate)::value>(tmem, w, x, dhi, idesc);
#pragma unroll
                for (int k = 1; k < BK / 16; ++k) umma<CG, true>(tmem, w + 2 * k, x + 2 * k, dhi, idesc);
            };
            auto small_terms = [&](uint32_t w, auto accumulate) {
                const uint32_t x = w + 2 * W_BYTES / 16;
                umma<CG, decltype(accumulate)::value>(rest, w + W_BYTES / 16, x, dhi, idesc);
#pragma unroll
                for (int k = 1; k < BK / 16; ++k) umma<CG, true>(rest, w + W_BYTES / 16 + 2 * k, x + 2 * k, dhi, idesc);
#pragma unroll
                for (int k = 0; k < BK / 16; ++k) umma<CG, true>(rest, w + 2 * k, x + X_BYTES / 16 + 2 * k, dhi, idesc);
            };
            const std::integral_constant<bool, true> add;
            const std::integral_constant<bool, false> set;
            int s = 0;
            bool ok = true;
            for (int tile = group; tile < n_tiles && ok; tile += n_groups) {
                uint32_t held = 0, held_empty = 0;
                bool holds = false;
                for (int kb = 0, left = 0; kb < nst; ++kb) {
                    ok = wait_bar(full + 8 * s, ph, abort, a);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const bool begins = left == 0, ahead = begins && kb > 0;
                    if (begins) {
                        // the sums' place is read while the small terms of this stage and the one before run
                        left = min(kb == 0 ? FIRST : KGROUP, nst - kb);
                        if (ahead) small_terms(w, add);
                        ok = wait_bar(acc_empty, aph, abort, a);
                        if (!ok) break;
                        aph ^= 1;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        main_terms(set);
                    } else {
                        main_terms(add);
                    }
                    if (--left == 0) umma_commit<CG>(acc_full);
                    if (!ahead && (kb == 0 ? nst > 1 : kb == nst - 2 && kb > 1)) {
                        // a tile's first and last small terms come behind the main terms of two stages: the drain reads the small terms of
                        // the tile before, and the main terms of this one, meanwhile
                        held = w;
                        held_empty = empty + 8 * s;
                        holds = true;
                    } else {
                        const bool starts = kb == (nst > 1);
                        if (starts) {
                            ok = wait_bar(rest_empty, rph, abort, a);
                            if (!ok) break;
                            rph ^= 1;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        }
                        if (holds) {
                            if (starts) small_terms(held, set);
                            else small_terms(held, add);
                            umma_commit<CG>(held_empty);
                            holds = false;
                        }
                        if (kb == 0) small_terms(w, set);
                        else if (!ahead) small_terms(w, add);
                        umma_commit<CG>(empty + 8 * s);
                    }
                    if (kb == nst - 1) umma_commit<CG>(rest_full);
                    w += STAGE / 16;
                    if (++s == a.stages) { s = 0; ph ^= 1; w = (uint32_t)desc; }
                }
            }
        }
        leave();
        if (warp == MMA_WARP) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TMEM_COLS) : "memory");
            else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TMEM_COLS) : "memory");
        }
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    // -------------------------------------------------------------------- drain and finish
    const int quarter = warp & 3, part = warp >> 2;                                 // 32 TMEM lanes, a quarter of the columns
    const uint32_t taddr0 = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(part * CW);
    const int groups = 1 + (max(nst - FIRST, 0) + KGROUP - 1) / KGROUP;
    // the warp's columns from column `col` on, pair by pair, and the word that they are read
    auto take = [&](int col, uint32_t bar, auto put) {
        constexpr int LW = CW % 32 == 0 ? 32 : CW % 16 == 0 ? 16 : 8;
#pragma unroll
        for (int o = 0; o < CW; o += LW) {
            uint32_t r[LW];
            tmem_ld_n<LW>(taddr0 + (uint32_t)(col + o), r, 0);
            tmem_wait<LW>(r);
            if (o + LW == CW) {
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                if (lane == 0) mbar_arrive_cluster(bar);
            }
#pragma unroll
            for (int i = 0; i < LW / 2; ++i) put(o / 2 + i, pack2(r[2 * i], r[2 * i + 1]));
        }
    };
    uint32_t fph = 0, rph = 0;
    const bool quits = a.withhold == 2 && quarter == 1;                             // test hook: one warp of each part gives up alone
    if (quits && lane == 0) give_up(abort, a);
    for (int tile = group; tile < n_tiles; tile += n_groups) {
        uint64_t acc[CW / 2];
#pragma unroll
        for (int i = 0; i < CW / 2; ++i) acc[i] = 0;
        bool ok = !quits;
#pragma unroll 1
        for (int g = 0; g < groups && ok; ++g) {
            ok = __all_sync(0xffffffffu, wait_bar(acc_full, fph, abort, a));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            take(0, acc_empty_leader, [&](int i, uint64_t v) { add2(acc[i], v); });
            fph ^= 1;
        }
        ok = __all_sync(0xffffffffu, ok && wait_bar(rest_full, rph, abort, a));
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t share = pack2(__float_as_uint(1.0f / kRest), __float_as_uint(1.0f / kRest));
            take(REST, rest_empty_leader, [&](int i, uint64_t v) { fma2(acc[i], v, share); });
            rph ^= 1;
        }
        // behind the vote the records of the tile before are read, too
        if (MODE == OUT_SCORE) ok = all_of_128(1 + part, ok);
        if (!ok) break;
        const int n = (tile % tiles_n) * (128 * CG) + rank * 128 + quarter * 32 + lane;
        const int m0 = (tile / tiles_n) * NT + part * CW, left = a.M - m0;
        const bool real = n < a.N;
        const float bias = a.bias && real ? __ldg(a.bias + n) : 0.0f;
        if constexpr (MODE == OUT_SCORE) {
            // each warp reduces its 32 lanes per column, the four quarters meet in shared memory
            const int nq = n - lane;
            auto records = [&](auto w, const int c0) {
                constexpr int W = decltype(w)::value;
                score_records<W>([&](int i) { return ((i & 1) ? hi_f(acc[(c0 + i) / 2]) : lo_f(acc[(c0 + i) / 2])) * a.inv; }, lane, nq < a.N ? nq : 0x7fffffff - 64, real,
                                 m0 + c0, a.M, W, a.targets, a.tlogit, recs + quarter * NT + part * CW + c0);
            };
#pragma unroll
            for (int c0 = 0; c0 + 16 <= CW; c0 += 16) records(std::integral_constant<int, 16>(), c0);
            asm volatile("bar.sync %0, 128;" ::"r"(1 + part) : "memory");
            const int c = quarter * 32 + lane, m = m0 + c;
            const int t128 = (tile % tiles_n) * CG + rank, n128 = (a.N + 127) / 128;
            if (c < CW && m < a.M && t128 < n128) a.stats[(size_t)m * n128 + t128] = merge_records(recs + part * CW + c, NT);
        } else if constexpr (MODE == OUT_F32) {
            // the residual may be the output itself, so the compiler cannot move loads above the stores ahead of them: a batch
            // of them is asked for first
            constexpr int RB = CW < 16 ? CW : 16;                            // columns per batch
            float* y = a.y + (size_t)m0 * a.ldy + n;
            const float* rp = a.residual + (size_t)m0 * a.ldy + n;
            float mine[(CW + 31) / 32];                                              // lane l: 1 / scale of columns l, l + 32, ..
#pragma unroll
            for (int j = 0; j < (CW + 31) / 32; ++j) mine[j] = a.row_inv && 32 * j + lane < left ? __ldg(a.row_inv + m0 + 32 * j + lane) : a.inv;
#pragma unroll
            for (int o = 0; o < CW; o += RB) {
                if (o >= left) break;
                float res[RB];
#pragma unroll
                for (int i = 0; i < RB; ++i) {
                    res[i] = a.residual && real && o + i < left ? *rp : 0.0f;
                    rp += a.ldy;
                }
#pragma unroll
                for (int i = 0; i < RB; ++i) {
                    const float inv = __shfl_sync(0xffffffffu, mine[(o + i) / 32], (o + i) & 31);
                    float v = fmaf((i & 1) ? hi_f(acc[(o + i) / 2]) : lo_f(acc[(o + i) / 2]), inv, bias);
                    if (a.gelu) v = gelu_f(v);
                    if (a.residual) v = res[i] + v;
                    if (real && o + i < left) *y = v;
                    y += a.ldy;
                }
            }
        } else {
            // lanes (2i, 2i + 1) hold neighbouring columns of the output: after the trade the even lane owns row m of both, the
            // odd lane row m + 1, and a half warp writes one 64-byte run
            const int odd = lane & 1;
            size_t at = (size_t)(m0 + odd) * a.ldy + (n & ~1);
#pragma unroll
            for (int i = 0; i < CW / 2; ++i) {
                if (2 * i < left) {
                    float v0 = fmaf(lo_f(acc[i]), a.inv, bias), v1 = fmaf(hi_f(acc[i]), a.inv, bias);
                    uint32_t w[3];
                    if (MODE == OUT_GELU) {
                        uint32_t t[2];
                        split2_f16(gelu_f(v0) * a.out_scale, gelu_f(v1) * a.out_scale, a.out_lo, t);
                        w[0] = t[0]; w[1] = t[1];
                    } else if (a.out_scale != 0.0f) {
                        uint32_t t[2];
                        split2_f16(v0 * a.out_scale, v1 * a.out_scale, a.out_lo, t);
                        w[0] = t[0]; w[1] = t[1]; w[2] = 0;
                    } else if (a.yp[2]) {
                        split2<3>(v0, v1, w);
                    } else {
                        uint32_t t[2];
                        split2<2>(v0, v1, t);
                        w[0] = t[0]; w[1] = t[1]; w[2] = 0;
                    }
                    const uint32_t got = __shfl_xor_sync(0xffffffffu, __byte_perm(w[0], w[1], odd ? 0x5410 : 0x7632), 1);
                    const uint32_t o0 = __byte_perm(w[0], got, odd ? 0x3254 : 0x5410), o1 = __byte_perm(w[1], got, odd ? 0x3276 : 0x7610);
                    if (real && 2 * i + odd < left) {
                        *(uint32_t*)(a.yp[0] + at) = o0;
                        *(uint32_t*)(a.yp[1] + at) = o1;
                    }
                    if (MODE == OUT_PLANES && a.yp[2]) {
                        const uint32_t g2 = __shfl_xor_sync(0xffffffffu, w[2], 1);
                        if (real && 2 * i + odd < left) *(uint32_t*)(a.yp[2] + at) = __byte_perm(w[2], g2, odd ? 0x3276 : 0x5410);
                    }
                }
                at += 2 * (size_t)a.ldy;
            }
        }
    }
    leave();
}

// Rows of x as f16 planes, each scaled by a power of two that brings its largest element into [2^14, 2^15), and rows of a Q8_0
// matrix as exact f16 planes; a warp per row. norms: null, or two zeroed words: bits of the largest square norm of a weight row, and the
// complement of the bits of the smallest that is not 0.
__global__ void __launch_bounds__(256) f16_planes_kernel(const float* __restrict__ x, int M, int K, __half* __restrict__ xh, __half* __restrict__ xl,
                                                         float* __restrict__ row_inv, const QMat w, __half* __restrict__ wh,
                                                         __half* __restrict__ wl, unsigned* __restrict__ norms) {
    constexpr int HELD = 8;
    pdl_trigger();
    const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row < M) {
        const float4* src = (const float4*)(x + (size_t)row * K);
        const int units = K >> 2;
        float big = 0.0f;
        // NaN falls out of the maximum: such a row is NaN at any scale
        auto most = [&](const float4& v) { big = fmaxf(fmaxf(big, fmaxf(fabsf(v.x), fabsf(v.y))), fmaxf(fabsf(v.z), fabsf(v.w))); };
        float4 held[HELD];                                    // a lane's first units stay in registers
#pragma unroll
        for (int i = 0; i < HELD; ++i) held[i] = lane + 32 * i < units ? src[lane + 32 * i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < HELD; ++i) most(held[i]);
        for (int u = lane + 32 * HELD; u < units; u += 32) most(src[u]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
        // 2^(14 - exponent), its exponent kept where it and its inverse are normal numbers
        const int e = (int)(__float_as_uint(big) >> 23);
        const int se = big == 0.0f || e == 255 ? 127 : min(max(127 + 14 + 127 - e, 1), 253);
        const float s = __uint_as_float((uint32_t)se << 23);
        auto put = [&](int u, const float4& v) {
            uint32_t p[2], q[2];
            split2_f16(v.x * s, v.y * s, kRest, p);
            split2_f16(v.z * s, v.w * s, kRest, q);
            ((uint2*)(xh + (size_t)row * K))[u] = make_uint2(p[0], q[0]);
            ((uint2*)(xl + (size_t)row * K))[u] = make_uint2(p[1], q[1]);
        };
#pragma unroll
        for (int i = 0; i < HELD; ++i)
            if (lane + 32 * i < units) put(lane + 32 * i, held[i]);
        for (int u = lane + 32 * HELD; u < units; u += 32) put(u, src[u]);
        if (lane == 0) row_inv[row] = __uint_as_float((uint32_t)(254 - se) << 23);
        return;
    }
    const int n = row - M;
    if (n >= w.N) return;
    const uint4* q = (const uint4*)(w.qu + (size_t)n * w.K);
    const __half* d = w.d + (size_t)n * (w.K >> 5);
    float norm = 0.0f;
#pragma unroll 2
    for (int c = lane; c < w.K >> 4; c += 32) {
        const uint4 u = q[c];
        const __half2 d2 = __half2half2(d[c >> 1]);
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            // 0x6400 | u is 1024 + u in f16: less 1152 it is the level, exactly
            const uint32_t t = __byte_perm((&u.x)[i >> 1], 0x64646464u, (i & 1) ? 0x4342 : 0x4140);
            const __half2 lv = __hsub2(*(const __half2*)&t, __half2half2(__ushort_as_half((unsigned short)0x6480)));
            const __half2 h = __hmul2(lv, d2), r = __hmul2(__hfma2(lv, d2, __hneg2(h)), __float2half2_rn(kRest));   // the rounding's remainder, exactly
            hi[i] = *(const uint32_t*)&h;
            lo[i] = *(const uint32_t*)&r;
            if (norms) {
                const float2 f = __half22float2(h);
                norm = fmaf(f.x, f.x, fmaf(f.y, f.y, norm));
            }
        }
        uint4 *ph = (uint4*)(wh + (size_t)n * w.K) + 2 * c, *pl = (uint4*)(wl + (size_t)n * w.K) + 2 * c;
        ph[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        ph[1] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
        pl[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        pl[1] = make_uint4(lo[4], lo[5], lo[6], lo[7]);
    }
    if (norms) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) norm += __shfl_xor_sync(0xffffffffu, norm, o);
        if (lane == 0 && norm > 0.0f) {                                                // squares: the order of the bits is theirs
            atomicMax(norms, __float_as_uint(norm));
            atomicMax(norms + 1, ~__float_as_uint(norm));
        }
    }
}

// x [n] as f16 planes of out.scale times its values.
__global__ void __launch_bounds__(256) split_f16_kernel(const float4* __restrict__ x, uint2* __restrict__ hi, uint2* __restrict__ lo, float scale, float rest, size_t n4) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
        const float4 v = x[i];
        uint32_t p[2], q[2];
        split2_f16(v.x * scale, v.y * scale, rest, p);
        split2_f16(v.z * scale, v.w * scale, rest, q);
        hi[i] = make_uint2(p[0], q[0]);
        lo[i] = make_uint2(p[1], q[1]);
    }
}

namespace {

struct TileChoice { int cg, nt; };

// Tile shape by waves of tiles x (stages x the cycles of a stage + the epilogue behind the last). What a stage takes, by clock64 in
// the issuer: a pair with 64 rows 648, 128 rows 798, 192 rows 1165, 256 rows 1547 (the MMAs alone 384, 768, 1152, 1536), a single CTA with 32
// rows 951, where reading the weight operand is what counts. 128 rows are entered dearer than that: with several waves the card's
// power limit counts, and a narrow tile moves more bytes for the same sums (32768 x 768 x 2304: 255 us, 192 rows 239, 256 rows 242).
TileChoice choose_tile(int M, int N, int K, int mode, int sms) {
    TileChoice best = {2, 64};
    double best_cost = 1e30;
    const int nst = (K + BK - 1) / BK;
    auto consider = [&](int cg, int nt, double step) {
        const long tiles = (long)((N + 128 * cg - 1) / (128 * cg)) * ((M + nt - 1) / nt);
        const long slots = std::max(1, sms / cg);
        const double cost = (double)((tiles + slots - 1) / slots) * nst * step + 15.0 * nt;
        if (cost < best_cost) { best_cost = cost; best = {cg, nt}; }
    };
    if (mode != OUT_SCORE) consider(1, 32, 950.0);
    consider(2, 64, 650.0);
    consider(2, 128, 900.0);
    consider(2, 192, 1165.0);
    consider(2, 256, 1547.0);
    return best;
}

template <int CG, int CW, int MODE>
int launch_one(const CUtensorMap (&map)[4], F16Args a, int tiles, int sms, cudaStream_t st) {
    constexpr int NT = 4 * CW, STAGE = 2 * W_BYTES + 2 * (NT / CG) * BK * 2;
    constexpr int FIXED = 1024 /* alignment slack */ + BAR_BYTES + (MODE == OUT_SCORE ? 4 * NT * 16 : 0);
    constexpr int STAGES = (SMEM_LIMIT - FIXED) / STAGE < MAX_STAGES ? (SMEM_LIMIT - FIXED) / STAGE : MAX_STAGES;
    constexpr int SMEM = STAGES * STAGE + FIXED;
    static bool ready[64] = {};
    int dev = 0;
    FC_CUDA(cudaGetDevice(&dev));
    if (!ready[dev & 63]) {
        FC_CUDA(cudaFuncSetAttribute(gemm_f16_kernel<CG, CW, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        ready[dev & 63] = true;
    }
    a.stages = STAGES;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(std::min(tiles, sms / CG) * CG));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = SMEM;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CG;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    FC_CUDA(cudaLaunchKernelEx(&cfg, gemm_f16_kernel<CG, CW, MODE>, map[0], map[1], map[2], map[3], a));
    FC_LAUNCHED();
    return FC_OK;
}

template <int MODE>
int launch_f16(const F16Mat& w, const Planes& x, F16Args a, int M, cudaStream_t st) {
    static int sms[64] = {};
    int dev = 0;
    FC_CUDA(cudaGetDevice(&dev));
    if (dev >= 64) return fail(FC_E_ARG, "device %d out of range", dev);
    if (!sms[dev]) FC_CUDA(cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev));
    if (M <= 0) return FC_OK;
    if (x.n != 2 || x.scale == 0.0f || x.lo != kRest || !w.hi || w.K % 32) return fail(FC_E_SHAPE, "the f16 GEMM takes two f16 planes of either side and K %% 32 == 0 (K = %d)", w.K);
    const TileChoice t = choose_tile(M, w.N, w.K, MODE, sms[dev]);
    a.N = w.N; a.K = w.K; a.M = M;
    a.inv = 1.0f / x.scale;
    a.wait_cycles = g_debug.wait_cycles; a.withhold = g_debug.withhold;
    CUtensorMap map[4];
    FC_TRY(encode_plane(&map[0], w.hi, w.N, w.K, 128, true));
    FC_TRY(encode_plane(&map[1], w.lo, w.N, w.K, 128, true));
    FC_TRY(encode_plane(&map[2], x.p[0], M, w.K, t.nt / t.cg, true));
    FC_TRY(encode_plane(&map[3], x.p[1], M, w.K, t.nt / t.cg, true));
    const int tiles = ((w.N + 128 * t.cg - 1) / (128 * t.cg)) * ((M + t.nt - 1) / t.nt);
    if (t.cg == 2)
        return t.nt == 256 ? launch_one<2, 64, MODE>(map, a, tiles, sms[dev], st)
             : t.nt == 192 ? launch_one<2, 48, MODE>(map, a, tiles, sms[dev], st)
             : t.nt == 128 ? launch_one<2, 32, MODE>(map, a, tiles, sms[dev], st) : launch_one<2, 16, MODE>(map, a, tiles, sms[dev], st);
    if constexpr (MODE != OUT_SCORE) return launch_one<1, 8, MODE>(map, a, tiles, sms[dev], st);
    return fail(FC_E_SHAPE, "no scoring tile of %d rows", t.nt);
}

}  // namespace

// A call of its own pays for turning the weight into planes, 5 bytes a weight, and has no split of K for few rows. Us on this kernel
// (on the levels), back to back, for N = 512 / 1024 / 4096:
//     K = 1024    512 rows 16.6 / 18.5 / 24.8 (14.5 / 16.6 / 22.8)    768 rows 16.7 / 18.6 / 28.9 (16.6 / 20.2 / 35.1)
//     K = 2048    768 rows 26.8 / 26.8 / 45.3 (20.6 / 26.9 / 57.2)   1024 rows 26.9 / 26.8 / 55.3 (21.6 / 30.8 / 59.6)
//     K = 3072   1024 rows 36.8 / 36.8 / 77.9 (24.8 / 36.0 / 81.5)   1536 rows 35.1 / 43.2 / 103 (35.1 / 46.3 / 118)
//     K = 4096   1536 rows 45.3 / 53.7 / 140 (41.2 / 57.6 / 155)     2048 rows 51.6 / 57.7 / 185 (45.4 / 61.7 / 168)
// The line lies where most shapes have gone over. Near it this kernel may be the slower one by up to 25 % (small N, whose levels split K), and
// large N would gain by it from fewer rows on; where both are close its results are, which are five times nearer to 64 bits.
bool f16_rows(int K, int M) { return M >= 512 && M >= K / 2; }

int launch_f16_planes(const float* x, int M, int K, const Planes& out, float* row_inv, const QMat& w, const F16Mat& planes, unsigned* norms, cudaStream_t st) {
    if (K % 4 || w.K % 16) return fail(FC_E_SHAPE, "f16 planes: row lengths %d, %d", K, w.K);
    f16_planes_kernel<<<(M + w.N + 7) / 8, 256, 0, st>>>(x, M, K, (__half*)out.p[0], (__half*)out.p[1], row_inv, w, (__half*)planes.hi, (__half*)planes.lo,
                                                         norms);
    FC_LAUNCHED();
    return FC_OK;
}

int launch_split_f16(const float* x, const Planes& out, size_t n, cudaStream_t st) {
    if (n % 4 || out.n != 2 || out.scale == 0.0f) return fail(FC_E_SHAPE, "split_f16: %zu elements into %d planes", n, out.n);
    const size_t n4 = n / 4;
    split_f16_kernel<<<(int)std::max<size_t>(1, std::min<size_t>((n4 + 255) / 256, 148 * 8)), 256, 0, st>>>(
        (const float4*)x, (uint2*)out.p[0], (uint2*)out.p[1], out.scale, out.lo, n4);
    FC_LAUNCHED();
    return FC_OK;
}

int launch_gemm_f16(const F16Mat& w, const Planes& x, const float* row_inv, const float* bias, const float* residual, int epi, float* y, const Planes* yp,
                    int M, int ldy, int* status, cudaStream_t st) {
    F16Args a = {};
    a.bias = bias; a.residual = residual; a.gelu = epi == EPI_GELU; a.row_inv = row_inv; a.y = y; a.ldy = ldy; a.status = status;
    if (epi != EPI_NONE && epi != EPI_GELU) return fail(FC_E_ARG, "epilogue %d is not one of this entry's", epi);
    if (y) return launch_f16<OUT_F32>(w, x, a, M, st);
    if (!yp || (epi == EPI_GELU && yp->n != 2) || (w.N & 31) || (ldy & 7) || residual || row_inv || (epi == EPI_GELU && yp->scale == 0.0f) || (yp->scale != 0.0f && yp->n != 2))
        return fail(FC_E_SHAPE, "plane output needs N %% 32 == 0, ldy %% 8 == 0, bf16 planes or two f16 planes (behind GELU these) and no residual");
    for (int p = 0; p < yp->n; ++p) a.yp[p] = (uint16_t*)yp->p[p];
    a.out_scale = yp->scale; a.out_lo = yp->lo;
    return epi == EPI_GELU ? launch_f16<OUT_GELU>(w, x, a, M, st) : launch_f16<OUT_PLANES>(w, x, a, M, st);
}

int launch_gemm_f16_score(const F16Mat& w, const Planes& x, const int* targets, void* stats, float* tlogit, int M, int* status, cudaStream_t st) {
    if (!targets || !stats || !tlogit) return fail(FC_E_ARG, "the scoring epilogue needs targets, stats and tlogit");
    F16Args a = {};
    a.targets = targets; a.stats = (float4*)stats; a.tlogit = tlogit; a.status = status;
    return launch_f16<OUT_SCORE>(w, x, a, M, st);
}

}  // namespace fc
