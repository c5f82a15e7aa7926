// What the tensor-core GEMMs share: barriers with bounded waits, TMA loads, tcgen05 issue, commit and read-back.
#pragma once
#include <cuda.h>

#include "planes.cuh"

namespace fc {
namespace tc {

__device__ __forceinline__ uint32_t s32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// One thread of the warp, in a form the compiler knows to be one: what a lone thread computes behind it can stay in uniform
// registers, where tcgen05 and TMA instructions take their operands from (behind lane == 0 each of them is moved there first).
__device__ __forceinline__ bool elect_one() {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok));
    return ok != 0;
}
// Barriers are named by their 32-bit shared address: a generic pointer would be converted again at every use.
__device__ __forceinline__ void mbar_init(uint32_t b, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(bytes) : "memory");
}
// b: a shared::cluster address, this CTA's or a peer's.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t b) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(b) : "memory");
}
// Up to `tries` times: a thread that finds the phase incomplete is suspended by the hardware for a while (without a time
// hint: with one, the wait is a software loop around nanosleep). The loop is four instructions, since a dozen warps sit in
// such loops at any time and their polls compete with the drain warps for issue slots.
__device__ __forceinline__ bool mbar_poll(uint32_t b, uint32_t parity, int tries) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .s32 n;\n\t"
        "mov.s32 n, %3;\n"
        "POLL_%=:\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "@p bra DONE_%=;\n\t"
        "sub.s32 n, n, 1;\n\t"
        "setp.gt.s32 q, n, 0;\n\t"
        "@q bra POLL_%=;\n"
        "DONE_%=:\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(b), "r"(parity), "r"(tries) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_sleep(uint32_t b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(b), "r"(parity), "r"(1000u) : "memory");
    return ok != 0;
}
template <class Args>
__device__ __forceinline__ void give_up(volatile int* abort, const Args& a) {
    *abort = 1;
    atomicExch(a.status, FC_E_TIMEOUT);
}
// Bounded wait. Returns false (after raising the status word) when the budget runs out or another role of this CTA
// already gave up. SLEEP: for the producers, which wait most of the time and are stages ahead.
template <bool SLEEP = false, class Args>
__device__ __forceinline__ bool wait_bar(uint32_t b, uint32_t parity, volatile int* abort, const Args& a) {
    if (__builtin_expect(SLEEP ? mbar_sleep(b, parity) : mbar_poll(b, parity, 256), 1)) return true;
    const long long t0 = clock64();
    while (!(SLEEP ? mbar_sleep(b, parity) : mbar_poll(b, parity, 256))) {
        if (*abort) return false;
        if (clock64() - t0 > a.wait_cycles) {
            give_up(abort, a);
            return false;
        }
    }
    return true;
}
// Warps that meet at a named barrier (128 threads) go on together or not at all: a wait that ran out in one of them may have been
// completed for another. Every warp votes once per tile, whatever its own wait said.
__device__ __forceinline__ bool all_of_128(int barrier, bool ok) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %2, 0;\n\tbarrier.cta.red.and.pred p, %1, 128, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(r) : "r"(barrier), "r"((uint32_t)ok) : "memory");
    return r != 0;
}
// mbar: shared::cluster address of the barrier the bytes complete on; with CG = 2 it may be the pair's other CTA's.
template <int CG>
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t mbar) {
    if (CG == 2)
        asm volatile(
            "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
            ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(mbar) : "memory");
    else
        asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
            ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(mbar) : "memory");
}
// K-major, 128-byte swizzle: 8-row atoms of 1024 bytes (SBO = 64 x 16 B), descriptor version 1.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)64 << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}
template <int CG, bool ACCUMULATE>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint32_t alo, uint32_t blo, uint32_t dhi, uint32_t idesc) {
    if (CG == 2)
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
            "setp.ne.b32 p, %5, 0;\n\tmov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %4, p;\n\t}"
            ::"r"(tmem_d), "r"(alo), "r"(blo), "r"(dhi), "r"(idesc), "n"(ACCUMULATE ? 1 : 0) : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
            "setp.ne.b32 p, %5, 0;\n\tmov.b64 a, {%1, %3};\n\tmov.b64 b, {%2, %3};\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %4, p;\n\t}"
            ::"r"(tmem_d), "r"(alo), "r"(blo), "r"(dhi), "r"(idesc), "n"(ACCUMULATE ? 1 : 0) : "memory");
}
// Arrives on the barrier at this offset when the MMAs issued so far have retired (CG = 2: in both CTAs of the pair).
template <int CG>
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    if (CG == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                     ::"r"(bar), "h"((uint16_t)3) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// N consecutive columns of the warp's 32 lanes into r[o ..].
template <int N, int CW>
__device__ __forceinline__ void tmem_ld_n(uint32_t taddr, uint32_t (&r)[CW], const int o) {
    if (N == 8) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {"
            "%0, %1, %2, %3, %4, %5, %6, %7"
            "}, [%8];"
            : "=r"(r[o + 0]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7])
            : "r"(taddr) : "memory");
    }
    if (N == 16) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {"
            "%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15"
            "}, [%16];"
            : "=r"(r[o + 0]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7]),
              "=r"(r[o + 8]), "=r"(r[o + 9]), "=r"(r[o + 10]), "=r"(r[o + 11]), "=r"(r[o + 12]), "=r"(r[o + 13]), "=r"(r[o + 14]), "=r"(r[o + 15])
            : "r"(taddr) : "memory");
    }
    if (N == 32) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {"
            "%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
            "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31"
            "}, [%32];"
            : "=r"(r[o + 0]), "=r"(r[o + 1]), "=r"(r[o + 2]), "=r"(r[o + 3]), "=r"(r[o + 4]), "=r"(r[o + 5]), "=r"(r[o + 6]), "=r"(r[o + 7]),
              "=r"(r[o + 8]), "=r"(r[o + 9]), "=r"(r[o + 10]), "=r"(r[o + 11]), "=r"(r[o + 12]), "=r"(r[o + 13]), "=r"(r[o + 14]), "=r"(r[o + 15]),
              "=r"(r[o + 16]), "=r"(r[o + 17]), "=r"(r[o + 18]), "=r"(r[o + 19]), "=r"(r[o + 20]), "=r"(r[o + 21]), "=r"(r[o + 22]), "=r"(r[o + 23]),
              "=r"(r[o + 24]), "=r"(r[o + 25]), "=r"(r[o + 26]), "=r"(r[o + 27]), "=r"(r[o + 28]), "=r"(r[o + 29]), "=r"(r[o + 30]), "=r"(r[o + 31])
            : "r"(taddr) : "memory");
    }
}
template <int CW>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t (&r)[CW]) {
    tmem_ld_n<(CW >= 32 ? 32 : CW)>(taddr, r, 0);
    if (CW > 32) tmem_ld_n<(CW > 32 ? CW - 32 : 8)>(taddr + 32, r, 32);
}
// The registers pass through the wait (eight at a time), so that nothing that reads them can be scheduled ahead of it.
template <int CW>
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[CW]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < CW; i += 8)
        asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]), "+r"(r[i + 6]), "+r"(r[i + 7]));
}
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) { return (uint64_t)hi << 32 | lo; }
__device__ __forceinline__ float lo_f(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi_f(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ void fma2(uint64_t& acc, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float redux_max(float v) {
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float ex2(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// Softmax records of W activation rows (columns of a warp's tile), each over the warp's 32 weight rows: v(i) is the lane's logit of column i,
// of weight row n = n0 + lane (not real: beyond the matrix). rec[c] = (largest, sum of exp(logit - largest), first row that attains it);
// a target's own logit goes to tlogit. cols: columns that there are, rows of x from m0 on.
template <int W, class V>
__device__ __forceinline__ void score_records(V v, int lane, int n0, bool real, int m0, int M, int cols, const int* targets, float* tlogit, float4* rec) {
    const float kLog2e = 1.4426950408889634f;
    float e[W], my_max = -INFINITY;
    int my_idx = 0x7fffffff;
    const int col = lane & (W - 1);
    const int tgt = col < cols && m0 + col < M ? __ldg(targets + m0 + col) : -1;
    const uint32_t hits = __ballot_sync(0xffffffffu, tgt >= n0 && tgt < n0 + 32);
#pragma unroll
    for (int i = 0; i < W; ++i) {
        const float x = v(i);
        const float t = real ? x : -INFINITY;
        const float mx = redux_max(t);
        const uint32_t at = __ballot_sync(0xffffffffu, t == mx);
        e[i] = real ? ex2((x - mx) * kLog2e) : 0.0f;
        if (col == i) { my_max = mx; my_idx = n0 + __ffs(at) - 1; }
        if (hits >> i & 1) {                                                 // some lane's row is the target of column i
            const int tg = __shfl_sync(0xffffffffu, tgt, i);
            if (n0 + lane == tg) tlogit[m0 + i] = x;
        }
    }
    // transposing sum: W/2 + .. + 1 exchanges leave the lanes that agree in their low bits with parts of the sum of one column
#pragma unroll
    for (int o = W / 2; o > 0; o >>= 1) {
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const bool up = lane & o;
            const float keep = up ? e[i + o] : e[i], send = up ? e[i] : e[i + o];
            e[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (int o = W; o < 32; o <<= 1) e[0] += __shfl_xor_sync(0xffffffffu, e[0], o);
    if (lane < W && col < cols) rec[lane] = make_float4(my_max, e[0], __int_as_float(my_idx), 0.0f);
}
// The records of a column over the four quarters of 128 weight rows, `stride` apart.
__device__ __forceinline__ float4 merge_records(const float4* rec, int stride) {
    const float kLog2e = 1.4426950408889634f;
    float mx = -INFINITY, sum = 0.0f;
    int idx = 0x7fffffff;
#pragma unroll
    for (int q = 0; q < 4; ++q) mx = fmaxf(mx, rec[q * stride].x);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 r = rec[q * stride];
        if (r.x > -INFINITY || r.y != 0.0f) sum += r.y * ex2((r.x - mx) * kLog2e);
        if (r.x == mx) idx = min(idx, __float_as_int(r.z));
    }
    return make_float4(mx, sum, __int_as_float(idx), 0.0f);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// A [M][K] plane of 16-bit numbers through boxes of 64 columns x box_rows rows, 128-byte swizzle.
inline int encode_plane(CUtensorMap* map, const void* plane, int M, int K, int box_rows, bool f16) {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        FC_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
        if (!p || q != cudaDriverEntryPointSuccess) return fail(FC_E_CUDA, "cuTensorMapEncodeTiled is not available");
        fn = (EncodeTiledFn)p;
    }
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    const CUresult r = fn(map, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)plane, dims, strides, box, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(FC_E_CUDA, "cuTensorMapEncodeTiled failed (%d) for a [%d][%d] plane", (int)r, M, K);
    return FC_OK;
}

}  // namespace tc
}  // namespace fc
