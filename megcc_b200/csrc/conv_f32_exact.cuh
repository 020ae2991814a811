// A tile of the fp16-plane kernels (conv_f32_half.cu, conv_f32_patch.cu) from two tf32 planes: for operands
// that two scaled fp16 values do not hold (conv_f32_split.cuh). All threads of the CTA come here when the tiles
// in their turn are done; tensor memory and the tile area of shared memory are free then.
//
// The converter warps load 32 channels of one filter tap of 128 pixels and of
// the tile's filter rows by ordinary loads, split them (v = hi + lo, hi the nearest tf32 value) and write the
// four planes, 128-byte swizzle; three passes of tcgen05.mma kind::tf32 into accumulators of their own, which the
// epilogue warps add up in fp32. Two sets of planes and accumulators: the next step's loads are under way
// while the MMAs run. Bound by the latency of a step (loads, barrier, MMAs, one behind the other), a code
// path that ordinary data takes for one tile in thousands.
#pragma once
#include <stdint.h>

#include "conv_f32_epilogue.cuh"
#include "conv_f32_split.cuh"
#include "f32_internal.h"
#include "umma_ptx.cuh"

namespace mb200 {

// tiles of a CTA that can be put off: beyond these the kernels are not taken
constexpr int kExactTiles = 4096;

// A CTA's tiles that are put off: a bit for each of its tiles in turn, and whether there are any. The converters,
// who see an operand that does not fit, set it once a tile, without a branch. The epilogue does not ask: it
// stores what it has, and the tile is stored again at the end. (A question in front of its stores cost the
// 32-column kernel 10 %, 32 x 320 x 320, 16 -> 32: 388 -> 426 us. Hence a residual in the result's
// own place is not for these kernels.)
struct LateTiles {
    uint32_t bits[kExactTiles / 32], any;
};
__device__ __forceinline__ void put_tile_off_if(bool misfit, uint32_t late, uint32_t ordinal) {
    asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t"
            "@q red.relaxed.cta.shared::cta.or.b32 [%1], %2;\n\t@q st.shared.u32 [%3], 1;\n\t}" ::"r"((uint32_t)misfit),
            "r"(late + (ordinal >> 5) * 4), "r"(1u << (ordinal & 31)), "r"(late + kExactTiles / 8)
            : "memory");
}

struct ExactOperands {
    const float* src;
    long long src_pitch;
    int ic, ih, iw, sh, sw, base_h, base_w, taps, taps_w;
    // Weight of output channel o, tap t, channel c: w[o * w_row + (t * w_ic + c) * w_step], plus the same of
    // w_lo where there is one (w_step is 1 then)
    const float *w, *w_lo;
    long long w_row, w_step;
    int w_ic;
};

// host: ... of a ConvBias. weights: the filter's two tf32 planes, or, raw, a product's second operand [K][N]
inline ExactOperands conv_f32_exact_operands(
        const ConvF32Args& a, const float* src, const float* weights, bool raw) {
    const int icp = conv_f32_padded_ic(a.ic), taps = a.kh * a.kw;
    ExactOperands g;
    g.src = src;
    g.src_pitch = a.src_pitch;
    g.ic = a.ic;
    g.ih = a.ih;
    g.iw = a.iw;
    g.sh = a.sh;
    g.sw = a.sw;
    g.base_h = -a.ph;
    g.base_w = -a.pw;
    g.taps = taps;
    g.taps_w = a.kw;
    g.w = weights;
    g.w_lo = raw ? nullptr : weights + (size_t)a.oc * taps * icp;
    g.w_row = raw ? 1 : (long long)taps * icp;
    g.w_step = raw ? a.oc : 1;
    g.w_ic = raw ? a.ic : icp;
    return g;
}

// kind::tf32: fp32 accumulate, tf32 A and B, both K-major in shared memory
__device__ __forceinline__ void umma_tf32_ss(
        uint32_t leader, uint32_t tmem_d, uint32_t a, uint32_t b, uint32_t desc_hi, uint32_t idesc,
        uint32_t accumulate) {
    asm volatile(
            "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
            "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
            "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], da, db, %4, p;\n\t}" ::"r"(tmem_d),
            "r"(a), "r"(b), "r"(desc_hi), "r"(idesc), "r"(accumulate), "r"(leader)
            : "memory");
}

// four values -> the 16 bytes at the same place of the two planes
__device__ __forceinline__ void store_tf32_planes(uint8_t* hi_plane, uint8_t* lo_plane, uint32_t at, float4 v) {
    const float x[4] = {v.x, v.y, v.z, v.w};
    float h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        h[i] = __uint_as_float((__float_as_uint(x[i]) + 0x1000u) & 0xFFFFE000u);
        l[i] = __fsub_rn(x[i], h[i]);
    }
    *reinterpret_cast<float4*>(hi_plane + at) = make_float4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<float4*>(lo_plane + at) = make_float4(l[0], l[1], l[2], l[3]);
}

// One tile, BN columns from n0. `pixel`: row of the tile -> {image, output row and column, whether it is there}.
// `area`: 1024-byte aligned shared memory, (64 + BN / 2) KB. `steps`: steps of this CTA before, whose last
// two `bars` (one arrival each) stand for. False: a wait ran out, for every thread. (Every role goes through the
// steps by itself, with the same barriers: one loop for all would hold the sums and the loads in one thread's
// registers.)
struct ExactPixel {
    int img, y, x;
    bool there;
};
template <int BN, class Pixel>
__device__ __forceinline__ bool exact_tile(
        const ExactOperands& g, const F32Epilogue& e, const Pixel& pixel, int oh, int ow, int n0, uint8_t* area,
        uint32_t tmem_base, uint64_t* bars, uint32_t& steps, volatile int* abort_flag, int* status) {
    using namespace umma;
    constexpr int kBM = 128, kChunk = 32;
    constexpr int kAPlane = kBM * 128, kBPlane = BN * 128, kSet = 2 * kAPlane + 2 * kBPlane;
    static_assert(kBM * (BN + 1) * 4 <= 2 * kSet, "the sums take the planes' place");
    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    const int blocks = (g.ic + kChunk - 1) / kChunk, total = g.taps * blocks;
    float* sums = reinterpret_cast<float*>(area);
    bool ok = true;
    auto lost = [&] {  // (a barrier of all threads)
        const bool any = __syncthreads_or(!ok);
        if (!ok && !*abort_flag) {
            *abort_flag = 1;
            atomicExch(status, ERR_EPILOGUE_WAIT);
        }
        return any;
    };

    if (warp >= 10) {
        // ---- eight warps: operands to planes ----
        constexpr int kARows = kBM / 32, kBRows = BN / 32;  // rows of a thread, 32 apart
        const int unit = threadIdx.x & 7, row = (threadIdx.x >> 3) & 31;
        float4 a[kARows], b[kBRows];
        // where the rows' pixels lie, their filter rows, and the step to come
        const float* image[kARows];
        int y0[kARows], x0[kARows];
#pragma unroll
        for (int i = 0; i < kARows; ++i) {
            const ExactPixel px = pixel(row + 32 * i);
            image[i] = g.src + (size_t)px.img * g.ih * g.iw * g.src_pitch;
            y0[i] = px.there ? px.y * g.sh + g.base_h : -(1 << 30);  // (outside under every tap)
            x0[i] = px.x * g.sw + g.base_w;
        }
        const float* w[kBRows];
#pragma unroll
        for (int i = 0; i < kBRows; ++i)
            w[i] = n0 + row + 32 * i < e.oc ? g.w + (size_t)(n0 + row + 32 * i) * g.w_row : nullptr;
        const long long to_lo = g.w_lo - g.w;
        int fy = 0, fx = 0, c = unit * 4;
        long long wk = (long long)c * g.w_step;  // tap and channel among a filter row's weights
        auto fetch = [&]() {
#pragma unroll
            for (int i = 0; i < kARows; ++i) {
                const int y = y0[i] + fy, x = x0[i] + fx;
                a[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c < g.ic && (unsigned)y < (unsigned)g.ih && (unsigned)x < (unsigned)g.iw)
                    a[i] = *reinterpret_cast<const float4*>(image[i] + ((long long)y * g.iw + x) * g.src_pitch + c);
            }
#pragma unroll
            for (int i = 0; i < kBRows; ++i) {
                b[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (!w[i] || c >= g.w_ic)
                    continue;
                const float* at = w[i] + wk;
                if (g.w_lo) {  // (whole vectors: the planes are padded with zeros)
                    const float4 h = *reinterpret_cast<const float4*>(at);
                    const float4 l = *reinterpret_cast<const float4*>(at + to_lo);
                    b[i] = make_float4(h.x + l.x, h.y + l.y, h.z + l.z, h.w + l.w);
                } else {
                    b[i].x = at[0];
                    if (c + 1 < g.w_ic)
                        b[i].y = at[g.w_step];
                    if (c + 2 < g.w_ic)
                        b[i].z = at[2 * g.w_step];
                    if (c + 3 < g.w_ic)
                        b[i].w = at[3 * g.w_step];
                }
            }
            c += kChunk;
            wk += kChunk * g.w_step;
            if (c >= blocks * kChunk) {  // the next tap
                wk += (long long)(g.w_ic - blocks * kChunk) * g.w_step;
                c = unit * 4;
                if (++fx == g.taps_w) {
                    fx = 0;
                    ++fy;
                }
            }
        };
        fetch();
        for (int step = 0; step < total; ++step) {
            const uint32_t s = steps + (uint32_t)step;
            uint8_t* planes = area + (s & 1) * kSet;
            if (step >= 2)  // the MMAs over this set, two steps ago, have retired
                ok = ok && mbar_wait(&bars[s & 1], ((s >> 1) - 1) & 1u, abort_flag);
#pragma unroll
            for (int i = 0; i < kARows; ++i) {
                const int r = row + 32 * i;
                store_tf32_planes(planes, planes + kAPlane, (uint32_t)(r * 128 + ((unit ^ (r & 7)) << 4)), a[i]);
            }
#pragma unroll
            for (int i = 0; i < kBRows; ++i) {
                const int r = row + 32 * i;
                store_tf32_planes(planes + 2 * kAPlane, planes + 2 * kAPlane + kBPlane,
                                  (uint32_t)(r * 128 + ((unit ^ (r & 7)) << 4)), b[i]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            if (lost())
                return false;
            if (step + 1 < total)
                fetch();
        }
    } else if (warp >= 2) {
        // ---- eight warps: sums ----
        constexpr int kCols = BN / 2;
        const int col0 = ((warp - 2) >> 2) * kCols;
        float sum[kCols];
#pragma unroll
        for (int j = 0; j < kCols; ++j)
            sum[j] = 0.f;
        // (a step behind the MMAs: one more trip for the last)
        for (int step = 0; step <= total; ++step) {
            if (step < total && lost())
                return false;
            if (step == 0)
                continue;
            const uint32_t s = steps + (uint32_t)step - 1;
            ok = ok && mbar_wait(&bars[s & 1], (s >> 1) & 1u, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok)
                continue;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t ta = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (s & 1) * BN + (uint32_t)col0;
#pragma unroll
            for (int c = 0; c < kCols / 16; ++c) {
                uint32_t v[16];
                tmem_ld16(ta + 16 * c, v);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    sum[16 * c + j] = __fadd_rn(sum[16 * c + j], __uint_as_float(v[j]));
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        }
        // every MMA has retired: through shared memory, so that a warp's stores are runs of a row
        float* to = sums + ((warp & 3) * 32 + lane) * (BN + 1) + col0;
        if (ok) {
#pragma unroll
            for (int j = 0; j < kCols; ++j)
                to[j] = sum[j];
        }
    } else {
        // ---- the MMA issuer (warp 1), and one that keeps step ----
        const uint32_t leader = warp == 1 && elect_one() ? 1u : 0u;
        constexpr uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(BN >> 3) << 17) |
                                   ((uint32_t)(kBM >> 4) << 24);
        // 128-byte swizzled K-major rows: 8-row groups 1024 bytes apart
        constexpr uint32_t kDescHi = (1u << 14) | (2u << 29) | (1024 / 16);
        for (int step = 0; step < total; ++step) {
            if (lost())
                return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t set = (steps + (uint32_t)step) & 1;
            const uint32_t a_hi = ((smem_u32(area + set * kSet) & 0x3FFFFu) >> 4) | 1u << 16;
            const uint32_t a_lo = a_hi + kAPlane / 16, b_hi = a_hi + 2 * kAPlane / 16, b_lo = b_hi + kBPlane / 16;
            const uint32_t d = tmem_base + set * BN;
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // eight floats each; the small products first
                umma_tf32_ss(leader, d, a_lo + 2 * k, b_hi + 2 * k, kDescHi, idesc, k != 0);
                umma_tf32_ss(leader, d, a_hi + 2 * k, b_lo + 2 * k, kDescHi, idesc, 1);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k)
                umma_tf32_ss(leader, d, a_hi + 2 * k, b_hi + 2 * k, kDescHi, idesc, 1);
            umma_commit_if(leader, smem_u32(&bars[set]));
            __syncwarp();
        }
    }
    steps += (uint32_t)total;
    if (lost())
        return false;
    if (warp >= 2) {
        with_act(e.act, [&](auto act) {
#pragma unroll 1
            for (int i = (int)threadIdx.x - 64; i < kBM * BN; i += 512) {
                const int r = i / BN, ch = n0 + i % BN;
                const ExactPixel px = pixel(r);
                if (!px.there || ch >= e.oc)
                    continue;
                const size_t m = ((size_t)px.img * oh + px.y) * ow + px.x;
                float v = act_f32<decltype(act)::value>(sums[r * (BN + 1) + i % BN] + (e.bias ? e.bias[ch] : 0.f));
                if (e.z)
                    v += e.z[m * e.z_pitch + ch];
                e.dst[m * e.dst_pitch + ch] = v;
            }
        });
    }
    __syncthreads();  // before the next tile takes the area
    return true;
}

// ... all of the CTA's. Params: the kernel's, with `exact`, `ep`, `m_tiles`, `n_tiles`, `oh`, `ow`, `status` and
// pixel(tile).
template <int BN, class Params>
__device__ __forceinline__ void exact_tiles_here(
        const Params& p, const LateTiles* late, const ColumnStates* columns, uint8_t* area, uint32_t tmem_base,
        uint64_t* bars, volatile int* abort_flag) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t steps = 0;
    int i = 0;
    for (int tile = (int)blockIdx.x; tile < p.m_tiles * p.n_tiles; tile += (int)gridDim.x, ++i) {
        if ((late->bits[i >> 5] >> (i & 31) & 1u) == 0 && !columns->is_wide(tile % p.n_tiles))
            continue;
        if (!exact_tile<BN>(p.exact, p.ep, p.pixel(tile), p.oh, p.ow, tile % p.n_tiles * BN, area, tmem_base, bars,
                            steps, abort_flag, p.status))
            return;
    }
}
template <int BN, class Params>
__device__ __noinline__ void exact_tiles_called(
        const Params& p, const LateTiles* late, const ColumnStates* columns, uint8_t* area, uint32_t tmem_base,
        uint64_t* bars, volatile int* abort_flag) {
    exact_tiles_here<BN>(p, late, columns, area, tmem_base, bars, abort_flag);
}
// (A kernel's 96 registers a thread are all taken in its loops, and what is not there may still cost: in line the
// 64-column kernel gets 24 bytes of spills, 32 x 80 x 80, 64 -> 64 71 -> 76 us; called, the 128-column one got
// 260 and the 32-column one is 1.5 % slower.)
template <int BN, class Params>
__device__ __forceinline__ void exact_tiles(
        const Params& p, const LateTiles* late, const ColumnStates* columns, uint8_t* area, uint32_t tmem_base,
        uint64_t* bars, volatile int* abort_flag) {
    if constexpr (BN != 64)
        exact_tiles_here<BN>(p, late, columns, area, tmem_base, bars, abort_flag);
    else
        exact_tiles_called<BN>(p, late, columns, area, tmem_base, bars, abort_flag);
}

}  // namespace mb200
