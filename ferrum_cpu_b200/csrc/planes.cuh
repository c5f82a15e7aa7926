// Splitting f32 values into bf16 terms (the Planes of fc_common.cuh), shared by every kernel that feeds the tensor cores.
#pragma once
#include <cuda_bf16.h>

#include "fc_common.cuh"

namespace fc {

// Two f32 values -> their bf16 terms: w[p] = term p of (v0 | v1 << 16), each the rounding of what the terms before left.
// With three terms the sum is exact; an infinite value keeps its infinity in the first term and zeros after it.
template <int P>
__device__ __forceinline__ void split2(float v0, float v1, uint32_t (&w)[P]) {
#pragma unroll
    for (int p = 0; p < P; ++p) {
        const __nv_bfloat162 h = __float22bfloat162_rn(make_float2(v0, v1));
        w[p] = *(const uint32_t*)&h;
        if (p + 1 < P) {
            const float2 hf = __bfloat1622float2(h);
            v0 -= hf.x;
            v1 -= hf.y;
            if (P == 3) {
                v0 = v0 == v0 ? v0 : 0.0f;
                v1 = v1 == v1 ? v1 : 0.0f;
            }
        }
    }
}
// Two f32 values -> f16 hi, and the remainder times lo: v to 2^-23 of itself or 2^-25 / lo, whichever is more, below 65504.
__device__ __forceinline__ void split2_f16(float v0, float v1, float lo, uint32_t (&w)[2]) {
    const __half2 h = __floats2half2_rn(v0, v1);
    const float2 hf = __half22float2(h);
    const __half2 l = __floats2half2_rn((v0 - hf.x) * lo, (v1 - hf.y) * lo);
    w[0] = *(const uint32_t*)&h;
    w[1] = *(const uint32_t*)&l;
}
constexpr int F16X2 = -2;   // in the place of a number of planes: two f16 planes of out.scale times the value, the second times out.lo
template <int P>
__device__ __forceinline__ void store_planes(const Planes& out, size_t i, float v) {
    constexpr int N = P == F16X2 ? 2 : P;
    uint32_t w[N];
    if constexpr (P == F16X2) split2_f16(v * out.scale, 0.0f, out.lo, w);
    else split2<P>(v, 0.0f, w);
#pragma unroll
    for (int p = 0; p < N; ++p) ((uint16_t*)out.p[p])[i] = (uint16_t)w[p];
}
template <int P>
__device__ __forceinline__ void store_planes4(const Planes& out, size_t i4, float4 v) {   // elements 4 i4 .. 4 i4 + 3
    constexpr int N = P == F16X2 ? 2 : P;
    uint32_t a[N], b[N];
    if constexpr (P == F16X2) {
        split2_f16(v.x * out.scale, v.y * out.scale, out.lo, a);
        split2_f16(v.z * out.scale, v.w * out.scale, out.lo, b);
    } else {
        split2<P>(v.x, v.y, a);
        split2<P>(v.z, v.w, b);
    }
#pragma unroll
    for (int p = 0; p < N; ++p) ((uint2*)out.p[p])[i4] = make_uint2(a[p], b[p]);
}

}  // namespace fc
