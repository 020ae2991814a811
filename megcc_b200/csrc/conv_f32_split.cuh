// fp32 values as two scaled fp16 ones, for the kernels that multiply them so (conv_f32_half.cu, conv_f32_patch.cu):
//     v s = hi + 2^-12 lo,   hi = RN_f16(v s),   lo = RN_f16(2^12 (v s - hi))      (v s - hi is exact)
// s is a power of two that a pixel's 64 K elements share, or an output channel's whole filter: it brings the
// largest of them into [2^14, 2^15). The two values hold 22 bits as long as both are normal fp16 numbers or
// exact, that is from the largest down to 2^-15 times s^-1, 2^-29 of the largest; below, what is lost is 2^-37
// times s^-1 at most. (With lo in its own place and not 2^12 times up, 22 bits end at 2^-17 of the largest.)
// The MMAs take the 2^12 back as they go on from the small products to hi * hi (umma_f16_* with a shift).
//
// What does not fit is found and goes another way (conv_f32_exact.cuh):
//   * a weight that is not 0 and below 2^-30 of its channel's largest, or an infinite one: the channel is
//     WIDE, and the tiles of its columns are multiplied from tf32 planes;
//   * an activation below 2^-30 of the largest of its 64. Its error, 2^-51 of the largest, is nothing beside
//     the sum's terms where every weight is at least 2^-25 of its channel's largest: 64 such errors times the
//     largest weight are then 2^-20 of the one term of the largest activation. Of 1152 N(0,1) weights that is
//     so for all but one channel in 10^4. Where a channel has smaller weights or zeros (LOOSE), such a pixel
//     sends its tile the same way. N(0,1) activations: one in 10^9.
//   * a pixel whose largest is above 2^100 or below 2^-90 (not 0): sums and factors stay in the range of fp32
//     between these whatever the weights. Infinities are above, so they take the tf32 planes too.
// Hence no finite operands lose more than 2^-20 of the sum of the terms' magnitudes, and ordinary ones what the
// two tf32 planes of conv_f32.cu lose.
#pragma once
#include <stdint.h>

#include "f32_internal.h"
#include "umma_ptx.cuh"

namespace mb200 {

constexpr int kLoShift = 12;

// kind::f16 instruction descriptor: fp32 accumulate, fp16 A and B, both K-major
__host__ __device__ constexpr uint32_t umma_idesc_f16(int m, int n) {
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// ---- scaling and splitting ----
// The scale that brings values up to `largest` in magnitude into [2^14, 2^15), as an exponent field.
// (Infinities and NaNs get some finite scale; a filter's values all below 2^-98 are scaled by less than that.)
__device__ __forceinline__ uint32_t scale_field(float largest) {
    const uint32_t e = (__float_as_uint(largest) & 0x7FFFFFFFu) >> 23;
    return min(268u - e, 239u);
}
// An activation's values count 2^14 times too much beside those of the filter, whose factor undoes its
// own scale only down to [1, 2): the running sums are the activations times numbers below 2, the last
// multiplication is exact.
__device__ __forceinline__ float field_to_float(uint32_t field) { return __uint_as_float(field << 23); }
__device__ __forceinline__ uint32_t pixel_factor_field(uint32_t scale) { return 240u - scale; }

// ---- what fits ----
// A converter's view of its pixels' largest values over a tile, in three instructions each: all of them 0 or
// between 2^-90 and 2^100?
struct LargestValues {
    uint32_t top, bottom;  // (as bits, ordered like magnitudes; 0 counts as the largest for `bottom`)
    __device__ __forceinline__ void reset() {
        top = 0;
        bottom = 0xffffffffu;
    }
    __device__ __forceinline__ void take(float largest) {
        const uint32_t bits = __float_as_uint(largest);
        top = max(top, bits);
        bottom = min(bottom, bits - 1u);
    }
    __device__ __forceinline__ bool fit() const {
        constexpr uint32_t kTop = (127u + 100u) << 23, kBottom = (127u - 90u) << 23;
        return top <= kTop && bottom >= kBottom - 1u;
    }
};
// |v| as a number that orders magnitudes, 0 last
__device__ __forceinline__ uint32_t magnitude_0_last(float v) { return __float_as_uint(v) * 2u - 1u; }
// ... the least that fits beside a scale (of a pixel in range): 2^-16 over the scale
__device__ __forceinline__ uint32_t least_magnitude(uint32_t scale) { return ((238u - scale) << 24) - 1u; }

// An output channel's word: its factor (a power of two), and in its sign and last bit what its weights are like.
// `least` over all of them, `least_nonzero` over those that are not 0
// (kWideChannel: f32_internal.h)
constexpr uint32_t kLooseChannel = 1u;
__device__ __forceinline__ uint32_t channel_word(float largest, float least, float least_nonzero) {
    const uint32_t scale = scale_field(largest);
    const bool infinite = __float_as_uint(largest) >= 0x7F800000u;
    const bool wide = infinite || (largest > 0.f && __fmul_rn(least_nonzero, field_to_float(scale)) < 0x1p-16f);
    const bool loose = least < __fmul_rn(largest, 0x1p-25f);
    return (infinite ? 254u : 268u - scale) << 23 | (wide ? kWideChannel : 0u) | (loose ? kLooseChannel : 0u);
}
__device__ __forceinline__ float channel_factor(uint32_t word) { return __uint_as_float(word & 0x7F800000u); }

// Which tile columns have a wide or a loose channel (columns 64 apart share a bit: the tf32 planes are never
// wrong). In `strict` the converters see whether to look at the smallest values too. They do so until the epilogue
// warps, who have nothing to do at first, have been through the channels' words (a converter that waited for that
// added 1 us to a layer of one image).
struct ColumnStates {
    uint32_t strict[2], loose[2], wide[2];
    __device__ __forceinline__ void reset() {
        strict[0] = strict[1] = 0xffffffffu;
        loose[0] = loose[1] = wide[0] = wide[1] = 0;
    }
    __device__ __forceinline__ bool is_strict(int column) const {
        return (*(volatile const uint32_t*)&strict[column >> 5 & 1] >> (column & 31) & 1u) != 0;
    }
    __device__ __forceinline__ bool is_wide(int column) const {
        return (wide[column >> 5 & 1] >> (column & 31) & 1u) != 0;
    }
};
template <int THREADS, int BARRIER>
__device__ __forceinline__ void find_column_states(
        const float* words, int oc, int bn, int thread, ColumnStates* s, uint32_t* any_wide) {
#pragma unroll 4
    for (int o = thread; o < oc; o += THREADS) {
        const uint32_t word = __float_as_uint(__ldg(words + o));
        if (word & (kWideChannel | kLooseChannel)) {
            const int column = o / bn;
            if (word & kLooseChannel)
                atomicOr(&s->loose[column >> 5 & 1], 1u << (column & 31));
            if (word & kWideChannel) {
                atomicOr(&s->wide[column >> 5 & 1], 1u << (column & 31));
                *any_wide = 1;
            }
        }
    }
    asm volatile("bar.sync %0, %1;" ::"n"(BARRIER), "n"(THREADS) : "memory");
    if (thread < 2)
        *(volatile uint32_t*)&s->strict[thread] = *(volatile uint32_t*)&s->loose[thread];
}

// Two values times a power of two -> their fp16 pairs (x0 in the lower half). Every product and the difference
// are exact. PACKED: two values an instruction, which is the faster form in conv_f32_half.cu, whose converters
// are its longest chain (32 x 80 x 80, 128 -> 128 3x3: 209 -> 200 us), and the slower one in conv_f32_patch.cu
// (32 x 320 x 320, 16 -> 32: 396 -> 406).
template <bool PACKED>
struct SplitScale;
template <>
struct SplitScale<false> {
    float once, up;  // a power of two, and 2^12 times that
    __device__ __forceinline__ explicit SplitScale(uint32_t field)
        : once(field_to_float(field)), up(field_to_float(field + kLoShift)) {}
};
template <>
struct SplitScale<true> {
    uint64_t once, up;  // ... each twice
    static __device__ __forceinline__ uint64_t pair_of(float v) {
        uint64_t r;
        asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
        return r;
    }
    __device__ __forceinline__ explicit SplitScale(uint32_t field)
        : once(pair_of(field_to_float(field))), up(pair_of(field_to_float(field + kLoShift))) {}
};
__device__ __forceinline__ void split_f16(
        float x0, float x1, const SplitScale<false>& scale, uint32_t& hi, uint32_t& lo) {
    constexpr float kUp = (float)(1 << kLoShift);
    float h0, h1;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(__fmul_rn(x1, scale.once)), "f"(__fmul_rn(x0, scale.once)));
    asm("{\n\t.reg .b16 a, b;\n\tmov.b32 {a, b}, %2;\n\tcvt.f32.f16 %0, a;\n\tcvt.f32.f16 %1, b;\n\t}"
        : "=f"(h0), "=f"(h1)
        : "r"(hi));
    asm("cvt.rn.f16x2.f32 %0, %1, %2;"
        : "=r"(lo)
        : "f"(__fmaf_rn(h1, -kUp, __fmul_rn(x1, scale.up))), "f"(__fmaf_rn(h0, -kUp, __fmul_rn(x0, scale.up))));
}
__device__ __forceinline__ void split_f16(
        float x0, float x1, const SplitScale<true>& scale, uint32_t& hi, uint32_t& lo) {
    asm("{\n\t.reg .b64 x, v, h;\n\t.reg .f32 a, b;\n\t.reg .b16 p, q;\n\t"
        "mov.b64 x, {%2, %3};\n\t"
        "mul.rn.f32x2 v, x, %4;\n\t"
        "mov.b64 {a, b}, v;\n\t"
        "cvt.rn.f16x2.f32 %0, b, a;\n\t"
        "mov.b32 {p, q}, %0;\n\tcvt.f32.f16 a, p;\n\tcvt.f32.f16 b, q;\n\t"
        "mov.b64 h, {a, b};\n\t"
        "mul.rn.f32x2 v, x, %5;\n\t"
        "fma.rn.f32x2 v, h, %6, v;\n\t"
        "mov.b64 {a, b}, v;\n\t"
        "cvt.rn.f16x2.f32 %1, b, a;\n\t}"
        : "=&r"(hi), "=r"(lo)
        : "f"(x0), "f"(x1), "l"(scale.once), "l"(scale.up), "l"(0xC5800000C5800000ull));  // (-4096, -4096)
}

// the magnitudes of a channel's weights, over a block of 256 threads
struct Magnitudes {
    float largest, least, least_nonzero;
    static __device__ __forceinline__ Magnitudes none() {
        return Magnitudes{0.f, __uint_as_float(0x7F800000u), __uint_as_float(0x7F800000u)};
    }
    __device__ __forceinline__ void take(float v) {
        const float m = fabsf(v);
        largest = fmaxf(largest, m);
        least = fminf(least, m);
        if (m != 0.f)
            least_nonzero = fminf(least_nonzero, m);
    }
    __device__ __forceinline__ void take(const Magnitudes& o) {
        largest = fmaxf(largest, o.largest);
        least = fminf(least, o.least);
        least_nonzero = fminf(least_nonzero, o.least_nonzero);
    }
    __device__ __forceinline__ uint32_t word() const { return channel_word(largest, least, least_nonzero); }
};
__device__ __forceinline__ Magnitudes block_magnitudes(Magnitudes v, Magnitudes* shared) {
#pragma unroll
    for (int d = 16; d > 0; d /= 2) {
        Magnitudes o;
        o.largest = __shfl_xor_sync(0xffffffffu, v.largest, d);
        o.least = __shfl_xor_sync(0xffffffffu, v.least, d);
        o.least_nonzero = __shfl_xor_sync(0xffffffffu, v.least_nonzero, d);
        v.take(o);
    }
    if ((threadIdx.x & 31) == 0)
        shared[threadIdx.x >> 5] = v;
    __syncthreads();
    v = shared[0];
#pragma unroll
    for (int w = 1; w < 8; ++w)
        v.take(shared[w]);
    return v;
}

__device__ __forceinline__ void mbar_arrive_u32(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

}  // namespace mb200
