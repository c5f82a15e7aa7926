// Q8_0 GEMM on the 5th-generation tensor cores:
//     Y[M][N] = X[M][K] · dequant(W[N][K])ᵀ + bias (+GELU / SwiGLU) (+residual)
//
// Replaces ops::linear_forward (ferrum_core/src/ops.rs:233-256) for M >= 2 with the weight kept packed. A Q8_0 level
// is an 8-bit whole number and therefore exact in bf16, so the tensor core multiplies the LEVELS and the block scale is
// applied afterwards: every 32-wide k-block is accumulated on its own in TMEM, and the warps that read it back fold it
// into f32 registers with one fused multiply-add by the row's block scale. What is left to split is the activation:
//     2 planes (math mode FC_MATH_BF16X3): x = x1 + x2 to 2^-17 relative, two MMAs per step
//     3 planes (math mode FC_MATH_FP32):   x = x1 + x2 + x3 exactly (3 x 8 bits of significand), three MMAs per step
// The weight is exact in both, d·q is never rounded. Dequantising the weight to bf16 hi + lo planes instead needs three
// MMAs per step for 2-plane precision (and two weight planes in shared memory): measured on 32768 x 768 x 2304, that
// form ran at 338 TFLOP/s of algorithmic work.
//
// The weight tile is the M operand of the MMA (TMEM lane = weight row) and the activation rows are its N operand
// (TMEM column = activation row). A thread that drains TMEM thus needs ONE scale per k-block, its row's, and the number
// of activation rows per tile is free in steps of 16 or 32.
//
// One CTA per SM, 640 threads in five warpgroups (registers 160 / 160 / 56 / 56 / 40 a thread):
//   warps 0-7   drain: per k-block tcgen05.ld of their 32 lanes x half of the columns, f32x2 FMA into registers; after the
//               last k-block bias / GELU / SwiGLU / residual or the softmax records, and the stores
//   warps 8-15  weights: 32 levels of a row per thread, u8 -> bf16 (two logic operations and one packed add per pair),
//               stored in the swizzled K-major layout the tensor core reads. With four warps (64 levels a thread) a stage
//               took about 1600 cycles of latency, twice what the MMAs take
//   warp 16     TMA: the activation planes of the stage (64 k each)
//   warps 17-18 MMA issue, one for the even and one for the odd k-blocks; warp 17 owns the TMEM allocation (512 columns:
//               four k-block buffers of up to 128 activation rows or three of 160, enough to hide the two barrier hops
//               between a k-block's MMAs and its drain). What a k-block costs its issuer besides the MMAs (two barrier waits, a commit,
//               fetching the loop's instructions again) is about 500 cycles, as long as the MMAs themselves: one issuer
//               leaves the tensor pipe idle half of the time, two hide each other's.
// CG = 2: a pair of CTAs shares a tile (tcgen05 cta_group::2): each holds its 128 of 256 weight rows and half of the
// activation rows, so that the activation tile is read from L2 once for 256 weight rows and its operand reads from shared
// memory halve. Up to 160 rows a tile: 192 and 256 leave two buffers and more accumulators than the drain warps' registers
// hold beside their working set (32768 x 768 x 2304: 160 rows 354 us, 128 rows 388, 192 rows 376, 256 rows 467).
// CG = 1 takes small problems: the K range may be split over a cluster of up to 8 CTAs whose partial sums meet through
// distributed shared memory in rank order, so that a few activation rows still occupy the GPU and results stay
// reproducible.
//
// Every wait is bounded; a wait that runs out raises the status word and all roles leave, in whatever order they learn of it.
// Bound: weight bytes for a few rows, the drain for many (2·M·N·K algorithmic FLOP, planes x that executed). Measured with the
// split of X into planes (of the f32 form this replaced: CUDA-core FMA, 42 TFLOP/s):
//     32768 x 768 x 2304   2 planes 348 us = 334 TFLOP/s   3 planes 369 us = 314 TFLOP/s
//     32768 x 1024 x 4096  2 planes 746 us = 368 TFLOP/s   3 planes 791 us = 348 TFLOP/s
//     4096 x 1024 x 4096   2 planes 109 us (126 before)    3 planes 112 us (811 before)
// Half as many MMAs again cost 3 to 6 %: the tensor pipe is active 33 % (2 planes) and 49 % (3) of the cycles. Where the roles
// wait, in cycles by clock64 around the waits, 4096 x 1024 x 4096 in pair tiles of 160, 2 / 3 planes: a 64-wide stage takes about
// 1710 / 1795, its MMAs 640 / 960; an issuer waits 610 / 547 of it for an accumulator buffer and 254 / 268 for a stage, the TMA
// warp 1141 / 1115 and the converters 651 / 719 for a free stage. The drain spends 201 / 219 of the 733 / 767 cycles of a
// 32-wide k-block on its wait, which is about what a wait on a completed phase costs: it is the role the others wait for.
// Longer rows dilute the epilogue (193 cycles a k-block at K = 1024, 65 at 3072) and nothing else.
#include <algorithm>
#include <type_traits>

#include "pdl.cuh"
#include "tc.cuh"

namespace fc {

using namespace tc;

namespace {

constexpr int BK = 64;                                  // k per stage: two Q8_0 blocks, one 128-byte swizzle row of bf16
constexpr int Q_BYTES = 128 * BK * 2;                   // the CTA's weight tile of a stage
constexpr int DRAIN_WARPS = 8, DQ_WARPS = 8;
constexpr int TMA_WARP = DRAIN_WARPS + DQ_WARPS, MMA_WARP = TMA_WARP + 1;   // MMA_WARP and MMA_WARP + 1
constexpr int THREADS = 640;
constexpr int MAX_STAGES = 8;
constexpr int TMEM_COLS = 512, MAX_BUFS = 4;            // k-block buffers of 128 or 160 columns
constexpr int SCORE_BYTES = 4 * 128 * 16;               // per (32-row quarter, column) softmax records
// Block scales travel to the drain warps through a ring of their own: a stage is free again when its MMAs have retired, and
// the drain may be MAX_BUFS k-blocks behind those (two stages, three when it is in the middle of one).
constexpr int SCALE_BYTES = 128 * 4, SCALE_EXTRA = 3;   // per slot: a row's two f16 scales; slots beyond the stages
constexpr int SMEM_LIMIT = 227 * 1024;

enum Mode : int { OUT_F32 = 0, OUT_PLANES = 1, OUT_GELU = 2 /* planes, after GELU */, OUT_SWIGLU = 3, OUT_SCORE = 4 };

struct TcArgs {
    const uint8_t* qu; const __half* d; int N, K, N_pad, M;
    int nt;                   // activation rows of a tile
    int stages, stage_bytes;
    int bufs, acc_cols;       // TMEM buffers and their columns
    int ksplit;               // CTAs of a cluster that share the K range (CG = 1)
    const float* bias; const float* residual; int gelu;
    float* y; int ldy;        // OUT_F32
    uint16_t* yp[3];          // OUT_PLANES / OUT_GELU / OUT_SWIGLU: bf16 planes, ldy elements apart
    // OUT_SCORE: per (row, 128-column tile) softmax statistics instead of the product (see launch_gemm_q8_tc_score)
    const int* targets; float4* stats; float* tlogit;
    int* status;
    long long wait_cycles;    // budget of every mbarrier wait
    int withhold;             // test hooks. 1: the TMA producer issues nothing, so the waits on its stages run out
};

// Barriers and flags at the end of the shared memory, by byte offset.
constexpr int BAR_FULL = 0, BAR_EMPTY = BAR_FULL + 8 * MAX_STAGES, BAR_ACC_FULL = BAR_EMPTY + 8 * MAX_STAGES, BAR_ACC_EMPTY = BAR_ACC_FULL + 8 * MAX_BUFS;
constexpr int BAR_TMEM = BAR_ACC_EMPTY + 8 * MAX_BUFS, BAR_ABORT = BAR_TMEM + 4, BAR_BYTES = BAR_ABORT + 4;

// Finishes neighbouring activation rows m, m + 1 of this thread's weight row n, two at a time from row m0 on. Called by
// whole warps whose lanes hold 32 consecutive n (plane outputs trade values between neighbouring lanes).
template <int P, int MODE>
struct Finish {
    const TcArgs& a;
    bool real, odd;
    float bias;
    size_t at;                // offset of (m, n) in the output (plane outputs: of the pair or row this lane stores)
    __device__ __forceinline__ Finish(const TcArgs& a_, int n, int lane, int m0) : a(a_), real(n < a_.N), odd(lane & 1) {
        bias = a.bias && real ? __ldg(a.bias + n) : 0.0f;
        at = MODE == OUT_F32 ? (size_t)m0 * a.ldy + n
                             : (size_t)(m0 + odd) * a.ldy + (MODE == OUT_SWIGLU ? n >> 1 : n & ~1);
    }
    // The residual of rows m + 2 i and m + 2 i + 1. Asked for ahead of a run of stores: the residual may be the output
    // itself, so the compiler cannot move the loads of the next pair above the stores of this one.
    __device__ __forceinline__ void residual(int i, int left, float& r0, float& r1) const {
        const float* r = a.residual + at + (size_t)(2 * i) * a.ldy;
        r0 = real && left > 0 ? r[0] : 0.0f;
        r1 = real && left > 1 ? r[a.ldy] : 0.0f;
    }
    // left: rows from m on that exist (at least 1); r0, r1: their residual
    __device__ __forceinline__ void operator()(int left, float v0, float v1, float r0 = 0.0f, float r1 = 0.0f) {
        v0 += bias;
        v1 += bias;
        if (MODE == OUT_GELU) { v0 = gelu_f(v0); v1 = gelu_f(v1); }
        if (MODE == OUT_F32) {
            if (a.gelu) { v0 = gelu_f(v0); v1 = gelu_f(v1); }
            if (real) {
                float* y = a.y + at;
                if (a.residual) { v0 = r0 + v0; v1 = r1 + v1; }
                y[0] = v0;
                if (left > 1) y[a.ldy] = v1;
            }
        } else if (MODE == OUT_SWIGLU) {
            // rows (2j, 2j + 1) of the weight are (gate_j, up_j) (llm.rs:417-428): the even lane finishes row m, the odd
            // lane row m + 1, each with one value from its neighbour
            const float got = __shfl_xor_sync(0xffffffffu, odd ? v0 : v1, 1);
            const float g = odd ? got : v0, u = odd ? v1 : got;
            const float h = __fmul_rn(__fdiv_rn(g, __fadd_rn(1.0f, expf(-g))), u);
            if (real && (!odd || left > 1)) {
                uint32_t w[P];
                split2<P>(h, 0.0f, w);
#pragma unroll
                for (int p = 0; p < P; ++p) a.yp[p][at] = (uint16_t)w[p];
            }
        } else {
            // lanes (2i, 2i + 1) hold neighbouring columns: after the trade the even lane owns row m of both, the odd
            // lane row m + 1, and a half warp writes one 64-byte run
            uint32_t w[P], out[P];
            split2<P>(v0, v1, w);
            const uint32_t got = __shfl_xor_sync(0xffffffffu, __byte_perm(w[0], w[1], odd ? 0x5410 : 0x7632), 1);
            out[0] = __byte_perm(w[0], got, odd ? 0x3254 : 0x5410);
            out[1] = __byte_perm(w[1], got, odd ? 0x3276 : 0x7610);
            if (P == 3) {
                const uint32_t g2 = __shfl_xor_sync(0xffffffffu, w[P - 1], 1);
                out[P - 1] = __byte_perm(w[P - 1], g2, odd ? 0x3276 : 0x5410);
            }
            if (real && (!odd || left > 1)) {
#pragma unroll
                for (int p = 0; p < P; ++p) *(uint32_t*)(a.yp[p] + at) = out[p];
            }
        }
        at += 2 * (size_t)a.ldy;
    }
};

}  // namespace

// CW: columns a drain warp handles (its half of the nt columns, or more: what lies beyond its own is folded into registers
// that nothing stores): 32, 64 or 80, loaded in one or two parts. A compile-time number, and no more than 80: with a branch
// around each part, or with 128 columns, the compiler's moves and spills cost more than the larger tile saves.
template <int CG, int P, int MODE, int CW>
__global__ void __launch_bounds__(THREADS, 1)
gemm_q8_tc_kernel(const __grid_constant__ CUtensorMap map0, const __grid_constant__ CUtensorMap map1,
                  const __grid_constant__ CUtensorMap map2, const TcArgs a) {
    extern __shared__ unsigned char smem_raw[];
    // offsets, not casts, so that every access below is known to be to shared memory
    unsigned char* smem = smem_raw + ((1024 - (s32(smem_raw) & 1023)) & 1023);
    __half* scales = (__half*)(smem + a.stages * a.stage_bytes);                 // [stages + SCALE_EXTRA][128 rows]
    float4* recs = (float4*)((unsigned char*)scales + (a.stages + SCALE_EXTRA) * SCALE_BYTES);   // OUT_SCORE only
    unsigned char* tail = (unsigned char*)recs + (MODE == OUT_SCORE ? SCORE_BYTES : 0);
    volatile int* abort = (volatile int*)(tail + BAR_ABORT);
    const uint32_t sb = s32(smem), full = s32(tail) + BAR_FULL, empty = s32(tail) + BAR_EMPTY;
    const uint32_t acc_full = s32(tail) + BAR_ACC_FULL, acc_empty = s32(tail) + BAR_ACC_EMPTY;
    // the warp index through a shuffle: everything computed from it is then known to be the same for the whole warp and
    // stays out of the vector registers, of which the drain warps have none to spare
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int csize = CG == 2 ? 2 : a.ksplit;
    const int rank = CG == 2 || csize > 1 ? (int)(blockIdx.x % csize) : 0;          // rank in the cluster (clusters are 1-d)
    const int group = blockIdx.x / csize, n_groups = gridDim.x / csize;             // clusters take tiles in turn
    const int tiles_n = (a.N + 128 * CG - 1) / (128 * CG), tiles_m = (a.M + a.nt - 1) / a.nt;
    const int n_tiles = tiles_n * tiles_m;
    const int nb = a.K >> 5;                                                        // 32-wide k-blocks of a row
    const int nst = (nb + 1) >> 1;                                                  // 64-wide stages of a row
    // this CTA's share of the K range, in stages (all of it unless the cluster splits K)
    const int st0 = CG == 2 ? 0 : rank * nst / csize, st1 = CG == 2 ? nst : (rank + 1) * nst / csize;
    const int xr = a.nt / CG;                                                       // activation rows in this CTA's shared memory
    const bool leader = CG == 1 || rank == 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(full + 8 * s, 1 + DQ_WARPS * CG);
            mbar_init(empty + 8 * s, 2);
        }
        for (int b = 0; b < MAX_BUFS; ++b) {
            mbar_init(acc_full + 8 * b, 1);
            mbar_init(acc_empty + 8 * b, DRAIN_WARPS * CG);
        }
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMA_WARP) {   // the MMA warp owns the tensor memory allocation (with CG = 2 one warp of each CTA takes part)
        if (CG == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tail + BAR_TMEM)), "r"((uint32_t)TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s32(tail + BAR_TMEM)), "r"((uint32_t)TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (CG == 2 || csize > 1) {
        __syncwarp();
        cluster_sync();
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, *(volatile uint32_t*)(tail + BAR_TMEM), 0);
    pdl_wait();                                             // set up while the kernel ahead still ran
    pdl_trigger();

    // the barriers the pair's MMA issuers wait on are the leader's
    const uint32_t full_leader = CG == 2 ? mapa(full, 0) : full, acc_empty_leader = CG == 2 ? mapa(acc_empty, 0) : acc_empty;

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
        if (CG == 2 || csize > 1) cluster_sync();
        else asm volatile("bar.sync 0, %0;" ::"n"(THREADS) : "memory");
    };

    if (warp >= TMA_WARP) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        if (warp == TMA_WARP && a.withhold != 1 && elect_one()) {
            // ------------------------------------------------------------ TMA producer
            int s = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int tile = group; tile < n_tiles && ok; tile += n_groups) {
                const int m0 = (tile / tiles_n) * a.nt + (CG == 2 ? rank * xr : 0);
                for (int kb = st0; kb < st1; ++kb) {
                    ok = wait_bar<true>(empty + 8 * s, ph, abort, a);
                    if (!ok) break;
                    const uint32_t dst = sb + s * a.stage_bytes, bar = full_leader + 8 * s;
                    if (leader) mbar_expect_tx(full + 8 * s, (uint32_t)(CG * P * xr * 128));
                    tma_load_2d<CG>(dst, &map0, kb * BK, m0, bar);
                    tma_load_2d<CG>(dst + xr * 128, &map1, kb * BK, m0, bar);
                    if (P == 3) tma_load_2d<CG>(dst + 2 * xr * 128, &map2, kb * BK, m0, bar);
                    if (++s == a.stages) { s = 0; ph ^= 1; }
                }
            }
        } else if ((warp == MMA_WARP || warp == MMA_WARP + 1) && leader && elect_one()) {
            // ------------------------------------------------------------ MMA issuers
            const int h = warp - MMA_WARP;                          // the k-block of each stage that is this warp's
            // bf16 x bf16 -> f32, M = 128 (256 for the pair), N = nt, both operands K-major
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(a.nt >> 3) << 17) | ((uint32_t)(8 * CG) << 24);
            const uint64_t desc = smem_desc(sb + 64 * h);           // 32 k = 64 bytes
            const uint32_t dhi = (uint32_t)(desc >> 32), plane = (uint32_t)xr * 8;   // descriptors count 16 bytes
            const int total = (group < n_tiles ? (n_tiles - group + n_groups - 1) / n_groups : 0) * (st1 - st0);
            uint32_t x = (uint32_t)desc, ph = 0, aph = 1;
            int s = 0, kb = st0, buf = h;                           // buffers in k-block order over all tiles
            for (int it = 0; it < total; ++it) {
                const bool whole = 2 * kb + 1 < nb;
                if (h == 0 || whole) {
                    if (!wait_bar(acc_empty + 8 * buf, aph, abort, a)) break;
                    if (!wait_bar(full + 8 * s, ph, abort, a)) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t q = x + P * plane, acc = tmem + buf * a.acc_cols;
                    // the small terms first: they meet a small accumulator
                    umma<CG, false>(acc, q, x + (P - 1) * plane, dhi, idesc);
                    umma<CG, true>(acc, q + 2, x + (P - 1) * plane + 2, dhi, idesc);
#pragma unroll
                    for (int p = P - 2; p >= 0; --p) {
                        umma<CG, true>(acc, q, x + p * plane, dhi, idesc);
                        umma<CG, true>(acc, q + 2, x + p * plane + 2, dhi, idesc);
                    }
                    umma_commit<CG>(acc_full + 8 * buf);
                } else if (!wait_bar(full + 8 * s, ph, abort, a)) {
                    break;
                }
                umma_commit<CG>(empty + 8 * s);                      // frees the stage when both issuers' MMAs have retired
                x += (uint32_t)a.stage_bytes / 16;
                if (++s == a.stages) { s = 0; ph ^= 1; x = (uint32_t)desc; }
                if (++kb == st1) kb = st0;
                buf += whole ? 2 : 1;
                if (buf >= a.bufs) { buf -= a.bufs; aph ^= 1; }
            }
        }
        leave();
        if (csize > 1 && CG == 1) cluster_sync();
        if (warp == MMA_WARP) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (CG == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TMEM_COLS) : "memory");
            else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)TMEM_COLS) : "memory");
        }
    } else if (warp >= DRAIN_WARPS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        // ---------------------------------------------------------------- weight levels -> bf16
        const int row = (threadIdx.x - DRAIN_WARPS * 32) >> 1, hk = threadIdx.x & 1;  // weight row of the CTA's tile, half of its 64 levels
        int s = 0, slot = 0;
        uint32_t ph = 1;
        bool ok = true;
        for (int tile = group; tile < n_tiles && ok; tile += n_groups) {
            const int n = (tile % tiles_n) * (128 * CG) + (CG == 2 ? rank * 128 : 0) + row;
            const bool real = n < a.N_pad;
            const __half* dsrc = a.d + (size_t)(real ? n : 0) * nb;
            const uint4* src = (const uint4*)(a.qu + (size_t)(real ? n : 0) * a.K);
            const uint4 zero = make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u);   // biased zeros
            // two stages of levels and scales are under way at any time, in two sets of registers that take turns: with one
            // stage ahead, a stage could not come more often than an L2 round trip
            struct Row { uint4 q[2]; __half d; } ra, rb;
            ra.d = rb.d = __float2half(1.0f);                                       // a matrix of levels alone has no scales
            auto fetch = [&](Row& r, int kb) {
                const bool have = real && kb < st1 && 2 * kb + hk < nb;
                if (have && a.d) r.d = dsrc[2 * kb + hk];
#pragma unroll
                for (int i = 0; i < 2; ++i)
                    r.q[i] = have ? __ldg(src + (2 * kb + hk) * 2 + i) : make_uint4(0x80808080u, 0x80808080u, 0x80808080u, 0x80808080u);   // biased zeros
            };
            auto put = [&](Row& r, int kb) {
                ok = __all_sync(0xffffffffu, wait_bar<true>(empty + 8 * s, ph, abort, a));
                if (!ok) return;
                scales[slot * 256 + row * 2 + hk] = r.d;
                slot = slot == a.stages + SCALE_EXTRA - 1 ? 0 : slot + 1;
                unsigned char* dst = smem + s * a.stage_bytes + P * xr * 128 + row * 128;
#pragma unroll
                for (int c = 0; c < 4; ++c) {                                       // 16-byte chunk: 8 levels
                    const uint32_t w0 = (&r.q[c >> 1].x)[(c & 1) * 2], w1 = (&r.q[c >> 1].x)[(c & 1) * 2 + 1];
                    uint32_t o[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        // u = q + 128 in 16-bit lanes. bf16 has 7 stored bits: 0x4300 | (u & 127) is 128 + (u & 127), and
                        // bit 7 of u turns -256 (0xC380) into -128 (0xC300), so that the sum is q, exactly
                        const uint32_t t = __byte_perm(i < 2 ? w0 : w1, 0, (i & 1) ? 0x4342 : 0x4140);
                        const uint32_t hi = (t & 0x007F007Fu) | 0x43004300u, sub = (t & 0x00800080u) ^ 0xC380C380u;
                        asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(o[i]) : "r"(hi), "r"(sub));
                    }
                    *(uint4*)(dst + (((hk * 4 + c) ^ (row & 7)) * 16)) = make_uint4(o[0], o[1], o[2], o[3]);   // 128-byte swizzle
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // generic writes -> tensor-core reads
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(full_leader + 8 * s);
                // after the fence: it waits for every load under way, new ones included (1400 cycles a stage with them)
                fetch(r, kb + 2);
                if (++s == a.stages) { s = 0; ph ^= 1; }
            };
            fetch(ra, st0);
            fetch(rb, st0 + 1);
            for (int kb = st0; kb < st1 && ok; kb += 2) {
                put(ra, kb);
                if (ok && kb + 1 < st1) put(rb, kb + 1);
            }
        }
        leave();
        if (csize > 1 && CG == 1) cluster_sync();
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 160;");
        // ---------------------------------------------------------------- drain and finish
        const int quarter = warp & 3, part = warp >> 2;                             // 32 TMEM lanes, half of the columns
        const int cw = a.nt >> 1;                                                   // columns of this warp (a multiple of 8)
        const uint32_t taddr0 = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(part * cw);
        const __half2* my_scale = (const __half2*)scales + quarter * 32 + lane;
        int slot = 0;
        uint32_t fph = 0;                                                           // phase of the acc_full barriers
        int buf = 0;
        const bool quits = a.withhold == 2 && quarter == 1;                         // test hook: one warp of each part gives up alone
        if (quits && lane == 0) give_up(abort, a);
        for (int tile = group; tile < n_tiles; tile += n_groups) {
            uint64_t acc[CW / 2];
#pragma unroll
            for (int i = 0; i < CW / 2; ++i) acc[i] = 0;
            bool ok = !quits;
            __half2 sc = __half2half2(__float2half(0.0f));
#pragma unroll 1
            for (int b = 2 * st0; b < min(2 * st1, nb) && ok; ++b) {
                ok = __all_sync(0xffffffffu, wait_bar(acc_full + 8 * buf, fph, abort, a));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                constexpr int LW = CW > 40 ? CW / 2 : CW;                                // columns of one load
                if (!(b & 1)) {
                    sc = my_scale[slot * 128];
                    slot = slot == a.stages + SCALE_EXTRA - 1 ? 0 : slot + 1;
                }
                const float scale = b & 1 ? __high2float(sc) : __low2float(sc);
                const uint64_t sc2 = pack2(__float_as_uint(scale), __float_as_uint(scale));
#pragma unroll
                for (int o = 0; o < CW; o += LW) {
                    uint32_t r[LW];
                    tmem_ld<LW>(taddr0 + (uint32_t)(buf * a.acc_cols + o), r);
                    tmem_wait<LW>(r);
                    if (o + LW == CW) {
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        if (lane == 0) mbar_arrive_cluster(acc_empty_leader + 8 * buf);
                    }
#pragma unroll
                    for (int i = 0; i < LW / 2; ++i) fma2(acc[o / 2 + i], pack2(r[2 * i], r[2 * i + 1]), sc2);
                }
                if (++buf == a.bufs) { buf = 0; fph ^= 1; }
            }
            // behind the vote the records of the tile before are read, too
            if (MODE == OUT_SCORE) ok = all_of_128(1 + part, ok);
            if (!ok) break;
            const int n = (tile % tiles_n) * (128 * CG) + (CG == 2 ? rank * 128 : 0) + quarter * 32 + lane;
            const int m0 = (tile / tiles_n) * a.nt + part * cw;
            if (CG == 1 && csize > 1) {
                // partial sums [column][128 rows] into the stage buffers: every MMA and copy of this CTA is done
                float* sum = (float*)smem + (size_t)(part * cw) * 128 + quarter * 32 + lane;
#pragma unroll
                for (int i = 0; i < CW / 2; ++i) {
                    if (2 * i < cw) {
                        sum[(2 * i) * 128] = lo_f(acc[i]);
                        sum[(2 * i + 1) * 128] = hi_f(acc[i]);
                    }
                }
            } else if (MODE == OUT_SCORE) {
                // softmax records of (activation row, 128 weight rows): each warp reduces its 32 lanes per column, the
                // four quarters meet in shared memory. Lane l ends up with column 32 j + l of its warp.
                const float kLog2e = 1.4426950408889634f;
                const bool real = n < a.N;
                const int nq = n - lane;
#pragma unroll
                for (int j = 0; j < CW / 32; ++j) {
                    float e[32], my_max = -INFINITY;
                    int my_idx = 0x7fffffff;
                    const int mt = m0 + j * 32 + lane;
                    const int tgt = j * 32 + lane < cw && mt < a.M ? __ldg(a.targets + mt) : -1;
                    const uint32_t hits = __ballot_sync(0xffffffffu, tgt >= nq && tgt < nq + 32);
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const float v = (i & 1) ? hi_f(acc[j * 16 + i / 2]) : lo_f(acc[j * 16 + i / 2]);
                        const float t = real ? v : -INFINITY;
                        const float mx = redux_max(t);
                        const uint32_t at = __ballot_sync(0xffffffffu, t == mx);
                        e[i] = real ? ex2((v - mx) * kLog2e) : 0.0f;
                        if (lane == i) { my_max = mx; my_idx = nq + __ffs(at) - 1; }
                        if (hits >> i & 1) {                                         // some lane's row is the target of column i
                            const int tg = __shfl_sync(0xffffffffu, tgt, i);
                            if (n == tg) a.tlogit[m0 + j * 32 + i] = v;
                        }
                    }
                    // transposing sum: 16 + 8 + 4 + 2 + 1 exchanges leave lane l with the sum of column l
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
                        for (int i = 0; i < o; ++i) {
                            const bool up = lane & o;
                            const float keep = up ? e[i + o] : e[i], send = up ? e[i] : e[i + o];
                            e[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                        }
                    }
                    if (j * 32 + lane < cw)
                        recs[quarter * 128 + part * cw + j * 32 + lane] = make_float4(my_max, e[0], __int_as_float(nq < a.N ? my_idx : 0x7fffffff), 0.0f);
                }
                asm volatile("bar.sync %0, 128;" ::"r"(1 + part) : "memory");
                const int c = quarter * 32 + lane, m = m0 + c;
                const int t128 = (tile % tiles_n) * CG + (CG == 2 ? rank : 0), n128 = (a.N + 127) / 128;
                if (c < cw && m < a.M && t128 < n128) {
                    float mx = -INFINITY, sum = 0.0f;
                    int idx = 0x7fffffff;
#pragma unroll
                    for (int q = 0; q < 4; ++q) mx = fmaxf(mx, recs[q * 128 + part * cw + c].x);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float4 r = recs[q * 128 + part * cw + c];
                        if (r.x > -INFINITY || r.y != 0.0f) sum += r.y * ex2((r.x - mx) * kLog2e);
                        if (r.x == mx) idx = min(idx, __float_as_int(r.z));
                    }
                    a.stats[(size_t)m * n128 + t128] = make_float4(mx, sum, __int_as_float(idx), 0.0f);
                }
            } else {
                const int left = a.M - m0;
                Finish<P, MODE> fin(a, n, lane, m0);
                if (MODE == OUT_F32 && a.residual) {
                    constexpr int RB = CW / 4;                                       // pairs per batch
#pragma unroll
                    for (int o = 0; o < CW / 2; o += RB) {
                        float r[2 * RB];
#pragma unroll
                        for (int i = 0; i < RB; ++i) fin.residual(i, min(cw, left) - 2 * (o + i), r[2 * i], r[2 * i + 1]);
#pragma unroll
                        for (int i = 0; i < RB; ++i)
                            if (2 * (o + i) < cw && 2 * (o + i) < left)
                                fin(left - 2 * (o + i), lo_f(acc[o + i]), hi_f(acc[o + i]), r[2 * i], r[2 * i + 1]);
                    }
                } else {
#pragma unroll
                    for (int i = 0; i < CW / 2; ++i)
                        if (2 * i < cw && 2 * i < left) fin(left - 2 * i, lo_f(acc[i]), hi_f(acc[i]));
                }
            }
        }
        leave();
        if (CG == 1 && csize > 1) {
            // every rank of the cluster finishes its share of the columns, adding the partial sums in rank order
            if (!*abort && group < n_tiles && MODE != OUT_SCORE) {
                const int tile = group;
                const int n = (tile % tiles_n) * 128 + quarter * 32 + lane, m0 = (tile / tiles_n) * a.nt;
                const int share = ((a.nt + csize - 1) / csize + 1) & ~1, c1 = min(a.nt, (rank + 1) * share);
                const uint32_t base = sb + (uint32_t)(quarter * 32 + lane) * 4;
                for (int c = rank * share + 2 * part; c < c1; c += 4) {
                    if (m0 + c >= a.M) break;
                    float v0 = 0.0f, v1 = 0.0f;
                    for (int r = 0; r < csize; ++r) {
                        const uint32_t at = mapa(base + (uint32_t)c * 512, r);
                        float p0, p1;
                        asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(p0) : "r"(at) : "memory");
                        asm volatile("ld.shared::cluster.f32 %0, [%1 + 512];" : "=f"(p1) : "r"(at) : "memory");
                        v0 += p0;
                        v1 += p1;
                    }
                    Finish<P, MODE> fin(a, n, lane, m0 + c);
                    float r0 = 0.0f, r1 = 0.0f;
                    if (MODE == OUT_F32 && a.residual) fin.residual(0, a.M - m0 - c, r0, r1);
                    fin(a.M - m0 - c, v0, v1, r0, r1);
                }
            }
            __syncwarp();
            cluster_sync();
        }
    }
}

// ------------------------------------------------------------------------------------------------ host side
namespace {
struct TileChoice { int cg, nt, ksplit; };

// Tile shape by a score in SM cycles: waves of tiles x (k-blocks x the slowest of the pipelines + what a tile costs once).
// Per 32-wide k-block: tensor pipe planes * nt; shared-memory bandwidth (128 bytes a cycle: operand reads of the MMAs, the
// TMA writes, the converted weights); the drain (tcgen05.ld and FMA, 32 lanes a cycle); the weight conversion. The score ranks
// shapes, it does not predict times: it counts throughputs, and what a k-block really takes is the latency of the drain's
// chain (wait, tcgen05.ld, FMA; see above): about 860 cycles with 160 rows where the score has 350 for two planes, 500 for three.
// split_k: the K range may be split over CTAs, which changes the order of the sums with the number of rows; callers whose
// results may not depend on how many rows share a launch leave it out.
TileChoice choose_tile(int M, int N, int K, int P, int mode, bool split_k, int sms) {
    TileChoice best = {1, 16, 1};
    double best_cost = 1e30;
    const int nst = (K + 63) / 64;
    auto consider = [&](int cg, int nt, int ks) {
        const long tiles = (long)((N + 128 * cg - 1) / (128 * cg)) * ((M + nt - 1) / nt);
        const long slots = sms / (cg * ks) < 1 ? 1 : sms / (cg * ks);
        if (ks > 1 && (tiles > slots || ks > nst)) return;            // a split-K cluster runs one tile
        const double waves = (double)((tiles + slots - 1) / slots);
        const double xr = (double)nt / cg;
        const double smem = (2.0 * P * (4096 + 32 * xr) + P * xr * 64 + 8192) / 128.0;
        const double step = std::max(std::max((double)P * nt, smem), std::max(1.3 * nt + 110.0, 190.0));
        const double steps = 2.0 * ((nst + ks - 1) / ks);
        const double once = (mode == OUT_SCORE ? 16.0 : 9.0) * nt + 400.0;
        const double cost = waves * (steps * step + once) + 2500.0 + (ks > 1 ? 1500.0 + 6.0 * nt : 0.0);
        if (cost < best_cost) { best_cost = cost; best = {cg, nt, ks}; }
    };
    for (int nt = 16; nt <= 128; nt += 16)
        for (int ks = 1; ks <= (split_k ? 8 : 1); ks *= 2) consider(1, nt, ks);
    if (M > 64)
        for (int nt = 64; nt <= (mode == OUT_SCORE ? 128 : 160); nt += 32) consider(2, nt, 1);   // records of 160 columns: 7 % slower head
    return best;
}

template <int CG, int P, int MODE, int CW>
int launch_one(const CUtensorMap (&map)[3], const TcArgs& a, int grid, int smem, cudaStream_t st) {
    static bool ready[64] = {};
    int dev = 0;
    FC_CUDA(cudaGetDevice(&dev));
    if (dev >= 64) return fail(FC_E_ARG, "device %d out of range", dev);
    if (!ready[dev]) {
        FC_CUDA(cudaFuncSetAttribute(gemm_q8_tc_kernel<CG, P, MODE, CW>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT));
        ready[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)(CG == 2 ? 2 : a.ksplit);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    FC_CUDA(cudaLaunchKernelEx(&cfg, gemm_q8_tc_kernel<CG, P, MODE, CW>, map[0], map[1], map[2], a));
    FC_LAUNCHED();
    return FC_OK;
}

template <int MODE>
int launch_tc(const QMat& w, const Planes& x, TcArgs a, int M, bool split_k, cudaStream_t st) {
    static int sms[64] = {};
    int dev = 0;
    FC_CUDA(cudaGetDevice(&dev));
    if (dev >= 64) return fail(FC_E_ARG, "device %d out of range", dev);
    if (!sms[dev]) FC_CUDA(cudaDeviceGetAttribute(&sms[dev], cudaDevAttrMultiProcessorCount, dev));
    if (M <= 0) return FC_OK;
    const int P = x.n;
    if ((P != 2 && P != 3) || w.K % 32) return fail(FC_E_SHAPE, "the tensor-core GEMM takes 2 or 3 planes and K %% 32 == 0 (got %d, %d)", P, w.K);
    const TileChoice t = choose_tile(M, w.N, w.K, P, MODE, split_k && MODE != OUT_SCORE, sms[dev]);
    a.qu = w.qu; a.d = w.d; a.N = w.N; a.K = w.K; a.N_pad = w.N_pad; a.M = M;
    a.nt = t.nt; a.ksplit = t.ksplit;
    a.acc_cols = t.nt > 128 ? 160 : 128;
    a.bufs = t.nt > 128 ? 3 : 4;
    const int xr = t.nt / t.cg;
    a.stage_bytes = P * xr * 128 + Q_BYTES;
    const int fixed = 1024 /* alignment slack */ + SCALE_EXTRA * SCALE_BYTES + BAR_BYTES + (MODE == OUT_SCORE ? SCORE_BYTES : 0);
    a.stages = std::min(MAX_STAGES, (SMEM_LIMIT - fixed) / (a.stage_bytes + SCALE_BYTES));
    a.wait_cycles = g_debug.wait_cycles; a.withhold = g_debug.withhold;
    CUtensorMap map[3];
    for (int p = 0; p < P; ++p) FC_TRY(encode_plane(&map[p], x.p[p], M, w.K, xr, false));
    if (P < 3) map[2] = map[1];
    const int tiles = ((w.N + 128 * t.cg - 1) / (128 * t.cg)) * ((M + t.nt - 1) / t.nt);
    const int csize = t.cg == 2 ? 2 : t.ksplit;
    const int grid = std::min(tiles, sms[dev] / csize) * csize;
    const int smem = a.stages * (a.stage_bytes + SCALE_BYTES) + fixed;
    auto go = [&](auto cg, auto cw) -> int {
        constexpr int CG = decltype(cg)::value, CW = decltype(cw)::value;
        return P == 2 ? launch_one<CG, 2, MODE, CW>(map, a, grid, smem, st) : launch_one<CG, 3, MODE, CW>(map, a, grid, smem, st);
    };
    const std::integral_constant<int, 1> one;
    const std::integral_constant<int, 2> two;
    const std::integral_constant<int, MODE == OUT_SCORE ? 64 : 32> ws;
    const std::integral_constant<int, 64> wm;
    const std::integral_constant<int, MODE == OUT_SCORE ? 64 : 80> wl;
    if (t.cg == 2) return t.nt > 128 ? go(two, wl) : t.nt > 64 ? go(two, wm) : go(two, ws);
    return t.nt > 64 ? go(one, wm) : go(one, ws);
}

template <int P>
__global__ void split_planes_kernel(const float* __restrict__ x, const float* __restrict__ cols, int k4, const Planes out, size_t n4) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += (size_t)gridDim.x * blockDim.x) {
        float4 v = ((const float4*)x)[i];
        if (cols) {
            const float4 s = ((const float4*)cols)[i % k4];
            v.x *= s.x; v.y *= s.y; v.z *= s.z; v.w *= s.w;
        }
        store_planes4<P>(out, i, v);
    }
}
}  // namespace

int launch_split_planes(const float* x, const Planes& out, size_t n, cudaStream_t st, const float* cols, int K) {
    if (n % 4 || (cols && K % 4)) return fail(FC_E_SHAPE, "split_planes: element count %zu is not a multiple of 4", n);
    const size_t n4 = n / 4;
    const int blocks = (int)std::max<size_t>(1, std::min<size_t>((n4 + 255) / 256, 148 * 8));
    if (out.n == 3) split_planes_kernel<3><<<blocks, 256, 0, st>>>(x, cols, K / 4, out, n4);
    else split_planes_kernel<2><<<blocks, 256, 0, st>>>(x, cols, K / 4, out, n4);
    FC_LAUNCHED();
    return FC_OK;
}

int launch_gemm_q8_tc(const QMat& w, const Planes& x, const float* bias, const float* residual, int epi, float* y, const Planes* yp,
                      int M, int ldy, int* status, cudaStream_t st, bool split_k) {
    TcArgs a = {};
    a.bias = bias; a.residual = residual; a.gelu = epi == EPI_GELU; a.y = y; a.ldy = ldy; a.status = status;
    if (yp) for (int p = 0; p < yp->n; ++p) a.yp[p] = (uint16_t*)yp->p[p];
    if (epi == EPI_SWIGLU) {
        if (y || !yp || yp->n != x.n || residual || (w.N & 1) || ldy < w.N / 2) return fail(FC_E_SHAPE, "the SwiGLU epilogue writes planes [M][N / 2]");
        return launch_tc<OUT_SWIGLU>(w, x, a, M, split_k, st);
    }
    if (epi != EPI_NONE && epi != EPI_GELU) return fail(FC_E_ARG, "epilogue %d is not one of this entry's", epi);
    if (y) return launch_tc<OUT_F32>(w, x, a, M, split_k, st);
    if (!yp || yp->n != x.n || (w.N & 31) || (ldy & 7) || residual)
        return fail(FC_E_SHAPE, "plane output needs N %% 32 == 0, ldy %% 8 == 0, as many planes as the input and no residual");
    return epi == EPI_GELU ? launch_tc<OUT_GELU>(w, x, a, M, split_k, st) : launch_tc<OUT_PLANES>(w, x, a, M, split_k, st);
}

int launch_gemm_q8_tc_score(const QMat& w, const Planes& x, const int* targets, void* stats, float* tlogit, int M, int* status,
                            cudaStream_t st) {
    if (!targets || !stats || !tlogit) return fail(FC_E_ARG, "the scoring epilogue needs targets, stats and tlogit");
    TcArgs a = {};
    a.targets = targets; a.stats = (float4*)stats; a.tlogit = tlogit; a.status = status;
    return launch_tc<OUT_SCORE>(w, x, a, M, false, st);
}

// scoring.rs:175-181 from the per-tile records of the fused head: a warp per row folds the records in tile
// order (lane l takes tiles l, l + 32, ...; the lanes are then merged pairwise in a fixed pattern), p =
// exp(target logit - max) / sum in f32, clamp_prob (loss.rs:12-18), ln in f64; greedy = the first column of the
// largest logit is the target.
__global__ void __launch_bounds__(256) score_combine_kernel(const float4* __restrict__ stats, const float* __restrict__ tlogit,
                                                            const int* __restrict__ targets, int M, int n_tiles, int V,
                                                            double* __restrict__ logprob, uint8_t* __restrict__ is_greedy) {
    const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= M) return;
    const int target = targets[row];
    if (target < 0 || target >= V) {
        if (lane == 0) { logprob[row] = 0.0; is_greedy[row] = 0; }
        return;
    }
    float m = -INFINITY, s = 0.0f;
    int idx = 0x7fffffff;
    auto merge = [&](float m2, float s2, int i2) {
        const float M2 = fmaxf(m, m2);
        const float f1 = m > -INFINITY ? expf(m - M2) : 0.0f, f2 = m2 > -INFINITY ? expf(m2 - M2) : 0.0f;
        s = s * f1 + s2 * f2;
        idx = m2 > m ? i2 : (m > m2 ? idx : min(idx, i2));
        m = M2;
    };
    const float4* rec = stats + (size_t)row * n_tiles;
    for (int t = lane; t < n_tiles; t += 32) {
        const float4 r = rec[t];
        merge(r.x, r.y, __float_as_int(r.z));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float m2 = __shfl_xor_sync(0xffffffffu, m, o), s2 = __shfl_xor_sync(0xffffffffu, s, o);
        const int i2 = __shfl_xor_sync(0xffffffffu, idx, o);
        // both lanes of a pair fold (lower lane, upper lane) in that order, so that they agree bit for bit
        if (lane & o) {
            const float m1 = m, s1 = s;
            const int i1 = idx;
            m = m2; s = s2; idx = i2;
            merge(m1, s1, i1);
        } else {
            merge(m2, s2, i2);
        }
    }
    if (lane == 0) {
        float p = expf(tlogit[row] - m) / s;
        if (p == p) p = fmaxf(p, 1e-12f);
        logprob[row] = log((double)p);
        is_greedy[row] = (uint8_t)(idx == target);
    }
}

int launch_score_combine(const void* stats, const float* tlogit, const int* targets, int M, int n_tiles, int V, double* logprob,
                         uint8_t* is_greedy, cudaStream_t st) {
    score_combine_kernel<<<(M + 7) / 8, 256, 0, st>>>((const float4*)stats, tlogit, targets, M, n_tiles, V, logprob, is_greedy);
    FC_LAUNCHED();
    return FC_OK;
}

}  // namespace fc

// =====================================================================================
// The allocation-free variant of the tensor-core linear
// =====================================================================================
// fc_q8_0_linear_dev needs scratch in global memory (the two bf16 planes the activations are
// split into, and a status word) and grows it with cudaMalloc. Here the same scratch is a
// file-scope device array of fixed size, so the call allocates nothing at all.
namespace {
constexpr size_t kStaticPlaneElems = (size_t)4 << 20;   // activations per call: M * K <= 4 Mi
// [hi plane | lo plane], 16 MiB per GPU that loads the library, held until the process exits.
static __device__ __align__(256) uint16_t g_noalloc_planes[2 * kStaticPlaneElems];
static __device__ __align__(256) int g_noalloc_status;

// Device addresses of the two arrays above, looked up once per device. In host code the names
// g_noalloc_planes / g_noalloc_status are only handles for cudaGetSymbolAddress: passing
// them to a kernel directly would hand it a host address.
struct NoAllocScratch {
    uint16_t* planes = nullptr;
    int* status = nullptr;
};
NoAllocScratch g_noalloc_dev[64];
}  // namespace

extern "C" int fc_q8_0_linear_dev_noalloc(const fc_qweight* w, const float* x_dev, const float* bias_dev, float* y_dev,
                                          int M, void* cuda_stream, int* timed_out) {
    using namespace fc;
    if (!w || !x_dev || !y_dev) return fail(FC_E_ARG, "fc_q8_0_linear_dev_noalloc: null argument");
    if (!aligned16(x_dev) || !aligned16(y_dev) || !aligned16(bias_dev))
        return fail(FC_E_ARG, "fc_q8_0_linear_dev_noalloc: x_dev, y_dev and bias_dev must be 16-byte aligned");
    if (M <= 0) return fail(FC_E_SHAPE, "fc_q8_0_linear_dev_noalloc: M = %d", M);
    int device = 0;
    const QMat* mat = qweight_matrix(w, &device);
    if (mat->K % 64) return fail(FC_E_SHAPE, "fc_q8_0_linear_dev_noalloc: K = %d is not a multiple of 64", mat->K);
    if ((size_t)M * mat->K > kStaticPlaneElems)
        return fail(FC_E_SHAPE, "fc_q8_0_linear_dev_noalloc: M * K = %zu exceeds the fixed scratch of %zu activations; "
                    "split the rows over several calls or use fc_q8_0_linear_dev", (size_t)M * mat->K, kStaticPlaneElems);
    if (device < 0 || device >= 64) return fail(FC_E_ARG, "fc_q8_0_linear_dev_noalloc: device %d out of range", device);
    FC_CUDA(cudaSetDevice(device));
    NoAllocScratch& sc = g_noalloc_dev[device];
    if (!sc.planes) {
        // set-up, first call on this device: resolve the device addresses of the static arrays
        void *p = nullptr, *s = nullptr;
        FC_CUDA(cudaGetSymbolAddress(&p, g_noalloc_planes));
        FC_CUDA(cudaGetSymbolAddress(&s, g_noalloc_status));
        sc.planes = (uint16_t*)p;
        sc.status = (int*)s;
    }
    cudaStream_t st = (cudaStream_t)cuda_stream;
    // the status word keeps whatever the previous call left in it: start from zero
    FC_CUDA(cudaMemsetAsync(sc.status, 0, sizeof(int), st));
    const Planes x = {{sc.planes, sc.planes + kStaticPlaneElems, nullptr}, 2};
    FC_TRY(launch_split_planes(x_dev, x, (size_t)M * mat->K, st));
    FC_TRY(launch_gemm_q8_tc(*mat, x, bias_dev, nullptr, EPI_NONE, y_dev, nullptr, M, mat->N, sc.status, st));
    if (timed_out) {
        FC_CUDA(cudaMemcpyAsync(timed_out, sc.status, sizeof(int), cudaMemcpyDeviceToHost, st));
        FC_CUDA(cudaStreamSynchronize(st));
        if (*timed_out != 0) return fail(FC_E_TIMEOUT, "a bounded wait inside the tensor-core GEMM ran out (status %d)", *timed_out);
    }
    return FC_OK;
}
