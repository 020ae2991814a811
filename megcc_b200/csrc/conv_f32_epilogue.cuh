// The epilogue that the fp32 tensor-core kernels share (conv_f32.cu, conv_f32_half.cu, conv_f32_patch.cu).
#pragma once
#include <stdint.h>

#include <type_traits>

#include "f32_internal.h"

namespace mb200 {

struct F32Epilogue {
    int oc, act;
    const float* bias;
    const float* z;  // optional tensor added after the activation (residual), or nullptr
    long long z_pitch;
    float* dst;
    long long dst_pitch;  // floats between consecutive pixels of dst (>= oc)
};

// 1 / (1 + 2^(-x log2 e)) from the hardware's two approximations (2 and 1 ulp), without the range
// handling that the general exponential and quotient put around them: a subnormal power is lost
// beside the 1 anyway, and an infinite one gives the right 0. 5 instructions instead of some 25.
__device__ __forceinline__ float sigmoid_f32(float x) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(x * -1.442695041f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
    return r;
}

template <int ACT>
__device__ __forceinline__ float act_f32(float x) {
    if (ACT == MB200_F32_RELU)
        return x > 0.f ? x : 0.f;
    if (ACT == MB200_F32_SIGMOID)
        return sigmoid_f32(x);
    if (ACT == MB200_F32_SILU)
        return x * sigmoid_f32(x);
    if (ACT == MB200_F32_H_SWISH) {
        float t = x + 3.f;
        t = t > 0.f ? t : 0.f;
        t = t > 6.f ? 6.f : t;
        return x * t * (1.f / 6.f);
    }
    return x;
}

// Calls f with the activation as a compile-time constant. The choice is made once per tile and
// warp: made per element (a run-time switch inside the unrolled loops) it serialised the
// elements, 250 clocks each, and the epilogue was the kernel's longest chain.
template <class F>
__device__ __forceinline__ void with_act(int act, F&& f) {
    switch (act) {
        case MB200_F32_RELU: f(std::integral_constant<int, MB200_F32_RELU>()); break;
        case MB200_F32_SIGMOID: f(std::integral_constant<int, MB200_F32_SIGMOID>()); break;
        case MB200_F32_SILU: f(std::integral_constant<int, MB200_F32_SILU>()); break;
        case MB200_F32_H_SWISH: f(std::integral_constant<int, MB200_F32_H_SWISH>()); break;
        default: f(std::integral_constant<int, MB200_F32_IDENTITY>()); break;
    }
}

// One pixel's channels of a finished tile (a row per lane): bias, activation, residual, stores.
// With a short K loop (1x1 filters) this is the kernel's longest chain. So the bias lies in
// shared memory (fetched once per tile column: from global memory each eight channels waited
// for their load behind the stores before them), the residual is brought into the L2 while the
// tile is computed, and stores are whole 32-byte sectors. 32 x 80 x 80 pixels of 128 channels to
// 80: 96 us before, 48 now (floor 26 by its bytes); 128 to 128: 66 -> 54. (Turning the tile round
// in shared memory, so that a warp stores 64-byte pieces of 16 rows instead of sectors of 32,
// measured the same within 3 % either way and costs 16 KB of the ring.)
template <int COLS, int ACT>
__device__ __forceinline__ void store_f32_row(
        const float (&sum)[COLS], const F32Epilogue& e, const float4* bias, size_t m, int ch0,
        bool vec4, bool vec8) {
    float* out = e.dst + m * e.dst_pitch + ch0;
    const float* zin = e.z ? e.z + m * e.z_pitch + ch0 : nullptr;
#pragma unroll
    for (int c = 0; c < COLS / 8; ++c) {
        if (ch0 + 8 * c >= e.oc)
            break;  // (also keeps the steps apart: run together they need too many registers)
        const bool whole = vec4 && ch0 + 8 * c + 8 <= e.oc;
        const float4 b0 = bias[2 * c], b1 = bias[2 * c + 1];
        const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j)
            v[j] = act_f32<ACT>(sum[8 * c + j] + b[j]);
        if (whole) {
            if (zin) {
                const float4 z0 = *(reinterpret_cast<const float4*>(zin) + 2 * c);
                const float4 z1 = *(reinterpret_cast<const float4*>(zin) + 2 * c + 1);
                v[0] += z0.x, v[1] += z0.y, v[2] += z0.z, v[3] += z0.w;
                v[4] += z1.x, v[5] += z1.y, v[6] += z1.z, v[7] += z1.w;
            }
            if (vec8) {
                asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(
                                     out + 8 * c),
                             "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]),
                             "f"(v[6]), "f"(v[7])
                             : "memory");
            } else {
                reinterpret_cast<float4*>(out)[2 * c] = make_float4(v[0], v[1], v[2], v[3]);
                reinterpret_cast<float4*>(out)[2 * c + 1] = make_float4(v[4], v[5], v[6], v[7]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (ch0 + 8 * c + j < e.oc)
                    out[8 * c + j] = zin ? v[j] + zin[8 * c + j] : v[j];
        }
    }
}

}  // namespace mb200
