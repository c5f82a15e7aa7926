// Upload-time repack of GGML Q8_0 blocks into the two device planes (levels, scales) of a QMat.
#include "fc_common.cuh"

namespace fc {

// ------------------------------------------------------------------------------- repack
// raw: N rows of K/32 blocks of 34 bytes. One thread per block.
__global__ void repack_q8_kernel(const uint8_t* __restrict__ raw, int N, int K, int N_pad,
                                 uint8_t* __restrict__ qu, __half* __restrict__ d, unsigned* top) {
    const int kb_per_row = K / 32;
    unsigned most = 0;
    const size_t total = (size_t)N_pad * kb_per_row;
    for (size_t b = (size_t)blockIdx.x * blockDim.x + threadIdx.x; b < total; b += (size_t)gridDim.x * blockDim.x) {
        const size_t row = b / kb_per_row;
        uint32_t w[8];
        __half scale = __ushort_as_half((unsigned short)0);
        if (row < (size_t)N) {
            const uint8_t* p = raw + b * 34;
            scale = __ushort_as_half((unsigned short)(p[0] | (p[1] << 8)));
            most = max(most, (unsigned)(p[0] | (p[1] << 8)) & 0x7fffu);
            // the 32 quants start 2 bytes into the block: only 2-byte aligned
            const uint16_t* p16 = (const uint16_t*)(p + 2);
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = ((uint32_t)p16[2 * i] | ((uint32_t)p16[2 * i + 1] << 16)) ^ 0x80808080u;
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) w[i] = 0x80808080u;
        }
        uint4* dst = (uint4*)(qu + b * 32);
        dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
        dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
        d[b] = scale;
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if ((threadIdx.x & 31) == 0 && most) atomicMax(top, most);
}

int launch_repack_q8(const uint8_t* raw, int N, int K, int N_pad, uint8_t* qu, __half* d, unsigned* top, cudaStream_t st) {
    const size_t total = (size_t)N_pad * (K / 32);
    const int threads = 256;
    const int blocks = (int)((total + threads - 1) / threads < 148 * 16 ? (total + threads - 1) / threads : 148 * 16);
    repack_q8_kernel<<<blocks, threads, 0, st>>>(raw, N, K, N_pad, qu, d, top);
    FC_LAUNCHED();
    return FC_OK;
}

}  // namespace fc
