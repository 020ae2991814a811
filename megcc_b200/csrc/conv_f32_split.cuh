// fp32 values as two scaled fp16 ones, for the kernels that multiply them so (conv_f32_half.cu, conv_f32_patch.cu).
#pragma once
#include <stdint.h>

#include "umma_ptx.cuh"

namespace mb200 {

// kind::f16 instruction descriptor: fp32 accumulate, fp16 A and B, both K-major
__host__ __device__ constexpr uint32_t umma_idesc_f16(int m, int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// ---- scaling and splitting ----
// The scale that brings values up to `largest` in magnitude into [2^14, 2^15), as an exponent field.
// (Infinities and NaNs get some finite scale and stay what they are; a filter's or pixel's values all below
// 2^-98 are scaled by less than that.)
__device__ __forceinline__ uint32_t scale_field(float largest) {
    const uint32_t e = (__float_as_uint(largest) & 0x7FFFFFFFu) >> 23;
    return min(268u - e, 239u);
}
// An activation's values count 2^14 times too much beside those of the filter, whose factor undoes its
// own scale only down to [1, 2): the product's sum then leaves the range of fp32 only where the
// sum of the activation times numbers of that size does.
__device__ __forceinline__ float field_to_float(uint32_t field) { return __uint_as_float(field << 23); }
__device__ __forceinline__ uint32_t pixel_factor_field(uint32_t scale) { return 240u - scale; }
__device__ __forceinline__ uint32_t channel_factor_field(uint32_t scale) { return 268u - scale; }

// two values times a power of two -> their fp16 pairs (x0 in the lower half)
__device__ __forceinline__ void split_f16(float x0, float x1, float scale, uint32_t& hi, uint32_t& lo) {
    float h0, h1;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(__fmul_rn(x1, scale)), "f"(__fmul_rn(x0, scale)));
    asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\tcvt.f32.f16 %0, a;\n\tcvt.f32.f16 %1, b;\n\t}"
        : "=f"(h0), "=f"(h1)
        : "r"(hi));
    // (exact: the scaled value and its rounding are less than a power of two apart)
    asm("cvt.rn.f16x2.f32 %0, %1, %2;"
        : "=r"(lo)
        : "f"(__fmaf_rn(x1, scale, -h1)), "f"(__fmaf_rn(x0, scale, -h0)));
}

// largest magnitude over a block of 256 threads
__device__ __forceinline__ float block_largest(float v, float* shared) {
#pragma unroll
    for (int d = 16; d > 0; d /= 2)
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, d));
    if ((threadIdx.x & 31) == 0)
        shared[threadIdx.x >> 5] = v;
    __syncthreads();
    v = shared[0];
#pragma unroll
    for (int w = 1; w < 8; ++w)
        v = fmaxf(v, shared[w]);
    return v;
}

__device__ __forceinline__ void mbar_arrive_u32(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

}  // namespace mb200
