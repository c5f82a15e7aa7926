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
template <int P>
__device__ __forceinline__ void store_planes(const Planes& out, size_t i, float v) {
    uint32_t w[P];
    split2<P>(v, 0.0f, w);
#pragma unroll
    for (int p = 0; p < P; ++p) ((uint16_t*)out.p[p])[i] = (uint16_t)w[p];
}
template <int P>
__device__ __forceinline__ void store_planes4(const Planes& out, size_t i4, float4 v) {   // elements 4 i4 .. 4 i4 + 3
    uint32_t a[P], b[P];
    split2<P>(v.x, v.y, a);
    split2<P>(v.z, v.w, b);
#pragma unroll
    for (int p = 0; p < P; ++p) ((uint2*)out.p[p])[i4] = make_uint2(a[p], b[p]);
}

}  // namespace fc
