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
// 80: 96 us before, 48 now (floor 26 by its bytes); 128 to 128: 66 -> 54. (For the narrow
// tiles of conv_f32.cu, which use this, turning the rows round as below is no gain: 32 x 160 x 160, 64 -> 32 1x1
// 63.8 -> 68.0 us, 32 x 320 x 320, 32 -> 64 3x3/2 204 -> 228; it costs the ring a stage.)
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

// A warp's rows (a pixel per lane), TURN columns at a time, turned round in shared memory, so that a warp's
// accesses to the result (and to z) are whole pieces of rows: a lane per row stored 32-byte sectors at the
// same place of 32 lines, which took the shared-memory pipe, that the MMAs read their operands by, three
// clocks each. Several rows are under way at a time: one by one they are a chain of 400 clocks each. 32 images of
// 80 x 80 (conv_f32_half.cu): 1x1 128 -> 128 58.8 -> 50.6 us, 128 -> 80 52.9 -> 44.3; 160 x 160, 3x3/2 64 -> 128
// 124 -> 117; 2048^3 product 63.7 -> 60.6. Halo patches, 320 x 320, 16 -> 32: 430 one by one, 370 now.
// `rows`: the pixel of the warp's first row, and for the row `first` (known at compile time) behind this lane's
// own first one whether it is there and its distance in pixels.
// FORM 0: whole 16-byte units, no z; 1: whole units and z; 2: any
template <int COLS, int TURN, int ACT, int FORM, bool SCALED, class Rows>
__device__ __forceinline__ void store_turned(
        const float (&sum)[COLS], const F32Epilogue& e, uint32_t buffer, const float* scales, const float* biases,
        const Rows& rows, int ch0) {
    constexpr int kUnits = TURN / 4;         // 16-byte units of a row
    constexpr int kRows = 32 / kUnits;       // rows of an access
    const int lane = threadIdx.x & 31;
    const int unit = lane % kUnits;
    // unit u of row r sits at unit u ^ swizzle(r): every eight lanes' accesses take all banks
    auto swizzle = [](int r) { return TURN == 32 ? r & 7 : r >> 1 & 3; };
    const int row0 = lane / kUnits;
    const size_t m0 = rows.first + row0;
    float* out0 = e.dst + m0 * e.dst_pitch + ch0 + unit * 4;
    const float* z0 = FORM != 0 && e.z ? e.z + m0 * e.z_pitch + ch0 + unit * 4 : nullptr;
#pragma unroll
    for (int c = 0; c < COLS / TURN; ++c) {
        const int ch = ch0 + c * TURN + unit * 4;
        if (ch0 + c * TURN >= e.oc)
            break;
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kUnits; ++u)
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(
                                 buffer + (lane * kUnits + (u ^ swizzle(lane))) * 16),
                         "f"(sum[c * TURN + 4 * u]), "f"(sum[c * TURN + 4 * u + 1]),
                         "f"(sum[c * TURN + 4 * u + 2]), "f"(sum[c * TURN + 4 * u + 3])
                         : "memory");
        __syncwarp();
        float4 scale = make_float4(1.f, 1.f, 1.f, 1.f);
        if (SCALED)
            scale = *reinterpret_cast<const float4*>(scales + c * TURN + unit * 4);
        const float4 bias = *reinterpret_cast<const float4*>(biases + c * TURN + unit * 4);
        constexpr int kAtOnce = FORM == 0 ? 4 : FORM == 1 ? 2 : 1;
#pragma unroll
        for (int h = 0; h < kUnits; h += kAtOnce) {
            float4 v[kAtOnce], add[kAtOnce];
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i) {
                const int r = (h + i) * kRows + lane / kUnits;
                asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(v[i].x), "=f"(v[i].y), "=f"(v[i].z), "=f"(v[i].w)
                             : "r"(buffer + (r * kUnits + (unit ^ swizzle(r))) * 16));
                if (FORM == 1) {
                    add[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (rows.there(row0, (h + i) * kRows) && ch < e.oc)
                        add[i] = *reinterpret_cast<const float4*>(z0 + rows.step((h + i) * kRows) * e.z_pitch + c * TURN);
                }
            }
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i) {
                // (the scale is a power of two: exact)
                v[i].x = act_f32<ACT>((SCALED ? __fmul_rn(v[i].x, scale.x) : v[i].x) + bias.x);
                v[i].y = act_f32<ACT>((SCALED ? __fmul_rn(v[i].y, scale.y) : v[i].y) + bias.y);
                v[i].z = act_f32<ACT>((SCALED ? __fmul_rn(v[i].z, scale.z) : v[i].z) + bias.z);
                v[i].w = act_f32<ACT>((SCALED ? __fmul_rn(v[i].w, scale.w) : v[i].w) + bias.w);
                if (FORM == 1)
                    v[i].x += add[i].x, v[i].y += add[i].y, v[i].z += add[i].z, v[i].w += add[i].w;
            }
#pragma unroll
            for (int i = 0; i < kAtOnce; ++i) {
                if (!rows.there(row0, (h + i) * kRows) || ch >= e.oc)
                    continue;
                float* out = out0 + rows.step((h + i) * kRows) * e.dst_pitch + c * TURN;
                if (FORM != 2) {
                    *reinterpret_cast<float4*>(out) = v[i];
                } else {
                    const float* z = z0 ? z0 + rows.step((h + i) * kRows) * e.z_pitch + c * TURN : nullptr;
                    out[0] = z ? v[i].x + z[0] : v[i].x;
                    if (ch + 1 < e.oc)
                        out[1] = z ? v[i].y + z[1] : v[i].y;
                    if (ch + 2 < e.oc)
                        out[2] = z ? v[i].z + z[2] : v[i].z;
                    if (ch + 3 < e.oc)
                        out[3] = z ? v[i].w + z[3] : v[i].w;
                }
            }
        }
    }
}

// ... with the activation and the form as compile-time constants
template <int COLS, int TURN, bool SCALED, class Rows>
__device__ __forceinline__ void store_f32_rows(
        const float (&sum)[COLS], const F32Epilogue& e, uint32_t buffer, const float* scales, const float* biases,
        const Rows& rows, int ch0) {
    const bool vec4 = ((e.dst_pitch | (e.z ? e.z_pitch : 0) | e.oc) & 3) == 0 &&
                      (((uintptr_t)e.dst | (uintptr_t)e.z) & 15) == 0;
    with_act(e.act, [&](auto a) {
        constexpr int kAct = decltype(a)::value;
        if (!vec4)
            store_turned<COLS, TURN, kAct, 2, SCALED>(sum, e, buffer, scales, biases, rows, ch0);
        else if (e.z)
            store_turned<COLS, TURN, kAct, 1, SCALED>(sum, e, buffer, scales, biases, rows, ch0);
        else
            store_turned<COLS, TURN, kAct, 0, SCALED>(sum, e, buffer, scales, biases, rows, ch0);
    });
}

// Rows that follow one another, up to `end`
struct F32RowsInLine {
    size_t first, end;
    __device__ __forceinline__ bool there(int row0, int row) const { return first + row0 + row < end; }
    __device__ __forceinline__ int step(int row) const { return row; }
};

}  // namespace mb200
