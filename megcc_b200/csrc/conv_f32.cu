// fp32 ConvBias / MatrixMul on the sm_100a tensor cores with fp32-level accuracy.
//
// tcgen05.mma kind::tf32 keeps 10 mantissa bits of each operand, which is not enough for the
// 1e-4 relative tolerance the fp32 path is held to (a single tf32 pass is off by ~5e-4 on
// N(0,1) data). Every operand is therefore split into two tf32 values,
//     v = hi + lo,   hi = RN_tf32(v),   lo = RN_tf32(v - hi)          (v - hi is exact)
// and the product is accumulated in the fp32 TMEM accumulator from three passes
//     hi*hi + lo*hi + hi*lo                                            (lo*lo is < 2^-22)
// which leaves a relative error of a few 2^-22 per product: the same order as fp32 itself.
// Both halves are exactly representable in tf32, so the result does not depend on how the
// tensor core treats the low 13 bits of its inputs.
//
// The tensor core adds each MMA's products into the TMEM accumulator with truncation, not
// round-to-nearest: every instruction pulls the running sum toward zero by about half an ulp.
// Over a long chain that is a SYSTEMATIC shrink of the result (measured: K = 1152 in one
// chain scaled outputs by 1 - 4e-6; through the 60 ConvBias layers between a detector's input
// and its heads that compounded to -3.6e-4, against a tolerance of 1e-4). Two measures keep
// the drift at the level of fp32 rounding:
//   * short chains: the K loop is cut into segments of eight K = 8 steps (with four the worst
//     error of a detector's heads is 0.15 of the tolerance and the kernel 10 % slower, with
//     sixteen 0.35, with thirty-two 0.6; eight leaves 0.23); every segment starts
//     fresh TMEM accumulators (two sets alternate) and the epilogue warps add the finished
//     segment into fp32 registers with round-to-nearest while the tensor core works on the
//     next one. A short partial sum is small against the final one and nearly uncorrelated
//     with its sign, so what is left of the drift largely cancels;
//   * the two correction passes (lo*hi, hi*lo) go to an accumulator of their own: they are
//     2^-11 of the main pass, so their truncation does not matter, and they no longer cause
//     two extra truncations of the main sum per step.
//
//   * filter: split once at load time (the Init step) into two K-major planes
//     [2][OC][KH][KW][IC];
//   * activation: fetched as it is by TMA (im2col, or tiled for a 1x1 filter) and split ON
//     CHIP: converter warps read each arrived fp32 tile, one pixel row per thread, and write its
//     hi and lo planes into TENSOR MEMORY, from where the MMAs take their A operand. What
//     bounds a tf32 contraction here is the SM's shared-memory port (128 bytes a clock): with
//     both operands in shared memory a 128 x 128 x 32 step moves 192 KB through it (TMA
//     writes, the converter's reads and its two plane writes, A and B reads of twelve MMAs),
//     1536 clocks against 768 of tensor time. With A in tensor memory 112 KB are left;
//   * accumulators. 128-column tiles: two main sets (segments alternate) and one correction
//     set per tile. The corrections are 2^-11 of the main sum, so one chain over the whole
//     tile is accurate enough, and the first correction MMA of a tile is issued behind the
//     tile's first main MMAs so that the wait for the previous tile's corrections to be
//     read is covered. 64 and 32 columns: main and correction columns lie side by side and
//     one MMA over the filter's two planes (2 BN columns) computes hi * [hi | lo] of both, so a
//     K step costs two instructions instead of three;
//   * a filter that fits shared memory beside a ring of A tiles stays resident (one tile
//     column, small K): the ring then carries activations only;
//   * few tiles (a small batch): the K loop is split over the CTAs of a cluster (2, 4 or 8), each
//     leaves its fp32 partial tile in its shared memory and finishes an equal share of the
//     rows, summing the partials over distributed shared memory in rank order (the result
//     does not depend on timing);
//   * structure of the kernel as in conv_umma.cu: persistent CTAs, warp 0 TMA producer, warp 1
//     MMA issuer and TMEM owner, warps 2..9 epilogue (tcgen05.ld -> + bias -> activation ->
//     optional residual add -> NHWC stores), warps 10..13 or 10..17 converters (one or two groups
//     of four), bounded waits.
//
// Replaces, for the fp32 configurations, the reference's im2col + 4x12 SIMD GEMM
// (compiler/lib/KernelGen/GeneralIntrinsic/ConvKernel/Fp32Im2col.cpp:122-217,
// GeneralIntrinsic/MatMulKernel/Fp32MatMulM4N12.cpp:8-160) and the SILU / SIGMOID elementwise
// kernel that follows a ConvBias in a YOLOX-style graph
// (BareMetal/ElemwiseKernel.cpp:52-53, BareMetal/Activation.cpp:31-37). Summation order
// differs from the reference's, as it does between any two fp32 GEMMs: parity is held to
// 1e-4 relative / 1e-5 absolute, not bit for bit.
#include <stdio.h>
#include <stdlib.h>

#include "conv_f32_epilogue.cuh"
#include "conv_f32_exact.cuh"
#include "f32_internal.h"
#include "pdl.h"
#include "tuning.h"
#include "umma_ptx.cuh"

namespace mb200 {

using namespace umma;

namespace {

constexpr int kBM = 128;
constexpr int kMaxStages = 8;

// kind::tf32 instruction descriptor: fp32 accumulate, tf32 A and B, both K-major
__host__ __device__ constexpr uint32_t umma_idesc_tf32(int m, int n) {
    return (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}

// A operand (fp32 bits, 10 mantissa bits used) in tensor memory, B in shared memory (descriptor as
// its two words); issued by the lane whose `leader` is non-zero
__device__ __forceinline__ void umma_tf32_ta(
        uint32_t leader, uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi,
        uint32_t idesc, uint32_t accumulate) {
    asm volatile(
            "{\n\t.reg .pred p, q;\n\t.reg .b64 d;\n\t"
            "mov.b64 d, {%2, %3};\n\t"
            "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], d, %4, p;\n\t}" ::"r"(tmem_d),
            "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(leader)
            : "memory");
}

// 16 columns of this warp's 32 TMEM lanes <- registers (complete after tcgen05.wait::st)
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
            "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
            "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
            "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
            "r"(v[15])
            : "memory");
}

// round to the nearest tf32 (ties to even): keeps sign, 8 exponent and 10 mantissa bits
__host__ __device__ inline float round_tf32(float v) {
    uint32_t u;
    memcpy(&u, &v, 4);
    u = (u + 0xFFFu + ((u >> 13) & 1u)) & 0xFFFFE000u;
    float r;
    memcpy(&r, &u, 4);
    return r;
}

// ------------------------------------------------------------------------------------------
// filter packing (load time)
// ------------------------------------------------------------------------------------------
// OIHW fp32 -> two K-major planes [2][OC][KH][KW][ICp] (hi, lo), ICp >= IC zero-filled. The lo
// plane holds the exact remainder (12 significant bits, the tensor core reads 11), so that
// hi + lo gives the weight back to the CUDA-core kernel.
__global__ void __launch_bounds__(256) pack_filter_f32_kernel(
        const float* __restrict__ src, float* __restrict__ dst, int oc, int ic, int icp, int kh,
        int kw) {
    const size_t plane = (size_t)oc * kh * kw * icp;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < plane;
         i += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % icp);
        size_t t = i / icp;
        const int fx = (int)(t % kw);
        t /= kw;
        const int fy = (int)(t % kh);
        const int o = (int)(t / kh);
        float v = 0.f;
        if (c < ic)
            v = src[(((size_t)o * ic + c) * kh + fy) * kw + fx];
        const float h = round_tf32(v);
        dst[i] = h;
        dst[plane + i] = __fsub_rn(v, h);
    }
}

// [K][N] fp32 (the second operand of a matrix product) -> the same two planes [2][N][Kp] in one
// pass: a 32 x 32 tile through shared memory, rows of 128 bytes read and written. Bound by HBM:
// 12 bytes per element.
__global__ void __launch_bounds__(256) pack_matrix_f32_kernel(
        const float* __restrict__ src, float* __restrict__ dst, int k, int n, int kp) {
    __shared__ float tile[32][33];
    const int n0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
    const size_t plane = (size_t)n * kp;
#pragma unroll
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int r = k0 + j, c = n0 + threadIdx.x;
        tile[j][threadIdx.x] = r < k && c < n ? __ldg(src + (size_t)r * n + c) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int c = n0 + j, r = k0 + threadIdx.x;
        if (c < n && r < kp) {
            const float v = tile[threadIdx.x][j];
            const float h = round_tf32(v);
            dst[(size_t)c * kp + r] = h;
            dst[plane + (size_t)c * kp + r] = __fsub_rn(v, h);
        }
    }
}

// ------------------------------------------------------------------------------------------
// the tensor-core kernel
// ------------------------------------------------------------------------------------------
struct F32ConvParams {
    int m_total, oc, oh, ow;
    int cblocks;  // row-sized channel blocks per tap
    int taps_w;
    int k_iters;
    int sh, sw, base_h, base_w;
    int m_tiles, n_tiles;
    int a_tiled;      // 1x1, stride 1, no padding: A is the plain matrix [pixels][channels]
    int b_lo_offset;  // rows from the hi plane to the lo plane of the filter
    int stages;       // depth of the shared-memory ring
    int b_resident;   // 1: the whole filter sits in front of the ring, stages hold A only
    int splits;       // CTAs of a cluster that share a tile's K loop (1: none)
    F32Epilogue ep;
    int* status;
    long long wait_cycles;
};

constexpr int kF32EpilogueWarps = 8;

template <int BN, int ROWB>
struct F32Cfg {
    static constexpr int kChans = ROWB / 4;  // floats per row = TMEM columns of an A plane
    static constexpr bool kWide = BN == 128;
    static constexpr int kAccCols = kWide ? 3 * BN : 4 * BN;
    static constexpr int kTRaw = (512 - kAccCols) / (2 * kChans);
    static constexpr int kTStages = kTRaw > 4 ? 4 : kTRaw;  // A stages in tensor memory
    static_assert(kTStages == 2 || kTStages == 4, "a whole number of turns of the converter groups");
    static constexpr int kSegIters = 256 / ROWB;  // stages per segment: eight K = 8 steps
    static constexpr int kABytes = kBM * ROWB;
    static constexpr int kBBytes = 2 * BN * ROWB;  // both planes of a filter tile
    static constexpr int kBarBytes = 1024;         // barriers, in front of everything
    // each epilogue warp's copy of its columns' bias, behind the barriers
    static constexpr int kBiasBytes = (kF32EpilogueWarps * BN / 2 * 4 + 1023) / 1024 * 1024;
    // shared memory for tiles: a CTA's 227 KB less alignment slack, barriers and bias
    static constexpr int kTileBudget = 227 * 1024 - 1024 - kBarBytes - kBiasBytes;
    static constexpr int kDynamic = kTileBudget + 1024 + kBarBytes + kBiasBytes;
    static constexpr int kPartPitch = BN + 4;      // floats per row of a split part's tile
};

// Eight epilogue warps, and one converter group of four warps for 128 columns (its epilogue holds
// 64 sums per thread: with 14 warps in the block a thread may have 128 registers), two groups
// that take turns for the narrower tiles, whose steps are shorter.
__host__ __device__ constexpr int f32_groups(int bn) { return bn == 128 ? 1 : 2; }
__host__ __device__ constexpr int f32_threads(int bn) {
    return 64 + 32 * kF32EpilogueWarps + 128 * f32_groups(bn);
}

// v = hi + lo: hi is v rounded to a tf32 value (ties away from zero), v - hi is exact and has
// at most 12 significant bits, of which the tensor core reads 11. Integer rounding: the
// conversion instruction runs at a fifth of the rate.
__device__ __forceinline__ void split_tf32(uint32_t v, uint32_t& hi, uint32_t& lo) {
    hi = (v + 0x1000u) & 0xFFFFE000u;
    lo = __float_as_uint(__fsub_rn(__uint_as_float(v), __uint_as_float(hi)));
}

template <int BN, int ROWB>
__global__ void __launch_bounds__(f32_threads(BN), 1) conv_f32_umma_kernel(
        const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
        const F32ConvParams p) {
    using C = F32Cfg<BN, ROWB>;
    constexpr int kChans = C::kChans;
    constexpr int kT = C::kTStages;
    constexpr int kTmemA = C::kAccCols;  // first column of the A stages
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full_bar = (uint64_t*)smem;             // [kMaxStages] TMA -> converters, MMA
    uint64_t* empty_bar = full_bar + kMaxStages;      // [kMaxStages]
    uint64_t* t_full = empty_bar + kMaxStages;        // [kT] converters -> MMA
    uint64_t* t_empty = t_full + 4;                   // [kT]
    uint64_t* acc_full = t_empty + 4;                 // [2]
    uint64_t* acc_empty = acc_full + 2;               // [2]
    uint64_t* corr_empty = acc_empty + 2;
    uint64_t* b_full = corr_empty + 1;
    uint64_t* drain_bar = b_full + 1;
    uint32_t* tmem_slot = (uint32_t*)(drain_bar + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    uint8_t* tiles = smem + C::kBarBytes + C::kBiasBytes;
    uint8_t* tiles_b = tiles;  // resident filter (if any), then the ring
    uint8_t* ring = tiles + (p.b_resident ? p.k_iters * C::kBBytes : 0);
    const int stage_bytes = C::kABytes + (p.b_resident ? 0 : C::kBBytes);

    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    const int total_tiles = p.m_tiles * p.n_tiles;
    // Work of this CTA. Split: one tile per cluster, a K range per CTA; else whole tiles, one
    // every gridDim.x.
    const int rank = p.splits > 1 ? (int)cluster_rank() : 0;
    const int first_tile = (int)blockIdx.x / p.splits;
    const int tile_step = p.splits > 1 ? total_tiles : (int)gridDim.x;
    const int my_tiles =
            first_tile < total_tiles ? (total_tiles - 1 - first_tile) / tile_step + 1 : 0;
    int kb = 0, ke = p.k_iters;
    if (p.splits > 1) {
        kb = (int)((long long)p.k_iters * rank / p.splits);
        ke = (int)((long long)p.k_iters * (rank + 1) / p.splits);
    }

    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxStages; ++s) {
            mbar_init(&full_bar[s], 1);
            // with a resident filter a stage is free once its converters have read it
            // (128 arrivals), otherwise once one of them has seen that the MMAs over it retired
            mbar_init(&empty_bar[s], p.b_resident ? 128 : 1);
        }
        for (int t = 0; t < kT; ++t) {
            mbar_init(&t_full[t], 128);
            mbar_init(&t_empty[t], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 32 * kF32EpilogueWarps);
        }
        mbar_init(corr_empty, 32 * kF32EpilogueWarps);
        mbar_init(b_full, 1);
        mbar_init(drain_bar, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    } else if (threadIdx.x == 32 * 2) {
        tma_prefetch_map(&map_a);
        tma_prefetch_map(&map_b);
    }
    if (warp == 1) {
        asm volatile(
                "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                        smem_u32(tmem_slot)),
                "r"(512)
                : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    auto give_up = [&](int code) {
        if (!*abort_flag) {
            *abort_flag = 1;
            atomicExch(p.status, code);
        }
    };

    if (warp == 0) {
        // ---------------- TMA producer (a converged warp, one lane issues) ----------------
        const uint32_t leader = elect_one() ? 1u : 0u;
        const uint32_t full_a = smem_u32(full_bar), empty_a = smem_u32(empty_bar);
        const uint32_t ring_a = smem_u32(ring);
        const int pixels = p.oh * p.ow;
        // where the first tile starts is worked out before the wait for the previous kernel
        int tile_n = first_tile % p.n_tiles, tile_m = first_tile / p.n_tiles;
        int img = tile_m * kBM / pixels;
        int rem = tile_m * kBM - img * pixels;
        int oy = rem / p.ow, ox = rem - oy * p.ow;
        int cb = 0, fx = 0, fy = 0;
        if (kb != 0) {  // a later part of a split tile starts inside the filter
            const int tap = kb / p.cblocks;
            cb = kb - tap * p.cblocks;
            fy = tap / p.taps_w;
            fx = tap - fy * p.taps_w;
        }
        pdl_wait();  // from here on the kernel touches global memory
        pdl_release();
        if (p.b_resident) {
            const uint32_t bar = smem_u32(b_full), b0 = smem_u32(tiles_b);
            mbar_expect_tx_if(leader, bar, (uint32_t)(p.k_iters * C::kBBytes));
            for (int it = 0; it < p.k_iters; ++it) {
                const uint32_t b = b0 + it * C::kBBytes;
                tma_load_2d_if(leader, b, &map_b, bar, it * kChans, 0);
                tma_load_2d_if(leader, b + C::kBBytes / 2, &map_b, bar, it * kChans, p.b_lo_offset);
            }
        }
        int s = 0;
        uint32_t parity = 1, slot = ring_a;
        bool ok = true;
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
            if (tile != first_tile) {
                tile_n = tile % p.n_tiles;
                tile_m = tile / p.n_tiles;
                img = tile_m * kBM / pixels;
                rem = tile_m * kBM - img * pixels;
                oy = rem / p.ow;
                ox = rem - oy * p.ow;
                cb = fx = fy = 0;
            }
            const int m0 = tile_m * kBM, n0 = tile_n * BN;
            const int base_w = ox * p.sw + p.base_w, base_h = oy * p.sh + p.base_h;
            for (int it = kb; it < ke; ++it) {
                ok = mbar_wait_u32(empty_a + 8 * s, parity, abort_flag, p.wait_cycles);
                if (!ok)
                    break;
                const uint32_t bar = full_a + 8 * s;
                mbar_expect_tx_if(leader, bar, (uint32_t)stage_bytes);
                if (p.a_tiled)
                    tma_load_2d_if(leader, slot, &map_a, bar, cb * kChans, m0);
                else
                    tma_load_im2col_4d_if(leader, slot, &map_a, bar, cb * kChans, base_w, base_h,
                                          img, (uint16_t)fx, (uint16_t)fy);
                if (!p.b_resident) {
                    const uint32_t b = slot + C::kABytes;
                    tma_load_2d_if(leader, b, &map_b, bar, it * kChans, n0);
                    tma_load_2d_if(leader, b + C::kBBytes / 2, &map_b, bar, it * kChans,
                                   n0 + p.b_lo_offset);
                }
                if (++cb == p.cblocks) {
                    cb = 0;
                    if (++fx == p.taps_w) {
                        fx = 0;
                        ++fy;
                    }
                }
                slot += (uint32_t)stage_bytes;
                if (++s == p.stages) {
                    s = 0;
                    slot = ring_a;
                    parity ^= 1u;
                }
            }
        }
        if (!ok)
            give_up(ERR_PRODUCER_WAIT);
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer (the whole warp waits, one lane issues) ----------------
        // The tensor pipe holds only a few MMAs beyond the one it executes, so every instruction
        // of this loop that is not an MMA shows as idle tensor time (a lone warp takes four to
        // six clocks for each). Hence: one segment per trip with its steps unrolled, descriptor
        // words and TMEM columns as running sums, one wait and one commit per step. The wait
        // for the converters covers the filter tile of the step too: they have waited for the
        // stage's TMA barrier before they arrived.
        const uint32_t leader = elect_one() ? 1u : 0u;
        constexpr uint32_t idesc = umma_idesc_tf32(kBM, BN);
        constexpr uint32_t idesc2 = umma_idesc_tf32(kBM, C::kWide ? BN : 2 * BN);
        // swizzled K-major tiles: 8-row groups 8 * ROWB bytes apart
        constexpr uint64_t kDesc = ((uint64_t)1 << 16) | ((uint64_t)(8 * ROWB / 16) << 32) |
                                   ((uint64_t)1 << 46) | ((uint64_t)(ROWB == 128 ? 2 : 4) << 61);
        constexpr uint32_t kDescHi = (uint32_t)(kDesc >> 32);
        constexpr int kSteps = ROWB / 32;          // K = 8 steps per stage
        constexpr int kSeg = C::kSegIters;         // stages per segment
        constexpr uint32_t kPlane = C::kBBytes / 2 / 16;
        const uint32_t t_full_a = smem_u32(t_full), t_empty_a = smem_u32(t_empty);
        const uint32_t acc_full_a = smem_u32(acc_full), acc_empty_a = smem_u32(acc_empty);
        const int k_len = ke - kb;
        // where the filter tiles lie: the ring's slots, or the resident filter's steps
        const int slots = p.b_resident ? k_len : p.stages;
        const uint32_t slot_step = (uint32_t)(p.b_resident ? C::kBBytes : stage_bytes) >> 4;
        const uint32_t b_first =
                (((p.b_resident ? smem_u32(tiles_b) : smem_u32(ring) + C::kABytes) & 0x3FFFFu) >> 4) |
                (uint32_t)kDesc;
        uint32_t b_lo = b_first;
        int slot = 0, t = 0;
        uint32_t t_parity = 0, tile_parity = 0, buf = 0, acc_parity = 1;
        bool ok = !p.b_resident || mbar_wait(b_full, 0, abort_flag, p.wait_cycles);
        for (int tile = 0; tile < my_tiles && ok; ++tile) {
            for (int left = k_len; left > 0; left -= kSeg) {
                ok = mbar_wait_u32(acc_empty_a + 8 * buf, acc_parity, abort_flag, p.wait_cycles);
                if (!ok)
                    break;
                const uint32_t tmem_d = tmem_base + buf * (C::kWide ? BN : 2 * BN);
                const uint32_t tmem_c = C::kWide ? tmem_base + 2 * BN : tmem_d + (uint32_t)BN;
#pragma unroll
                for (int j = 0; j < kSeg; ++j) {
                    if (j == 0 || j < left) {
                        ok = mbar_wait_u32(t_full_a + 8 * t, t_parity, abort_flag, p.wait_cycles);
                        if (!ok)
                            break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t a_hi = tmem_base + kTmemA + (uint32_t)(t * 2 * kChans);
                        const uint32_t a_lo = a_hi + kChans;
                        // a K step of 8 floats: 8 columns of A, 32 bytes inside B's swizzled row
                        // (+2 in the descriptor's 16-byte address units)
                        if constexpr (C::kWide) {
#pragma unroll
                            for (int k = 0; k < kSteps; ++k)
                                umma_tf32_ta(leader, tmem_d, a_hi + 8 * k, b_lo + 2 * k, kDescHi,
                                             idesc, (j | k) != 0);
                            if (j == 0 && left == k_len) {
                                // the previous tile's corrections must have been read
                                ok = mbar_wait(corr_empty, tile_parity ^ 1u, abort_flag,
                                               p.wait_cycles);
                                if (!ok)
                                    break;
                                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            }
#pragma unroll
                            for (int k = 0; k < kSteps; ++k) {
                                umma_tf32_ta(leader, tmem_c, a_lo + 8 * k, b_lo + 2 * k, kDescHi,
                                             idesc, (j | k) != 0 ? 1u : (left != k_len ? 1u : 0u));
                                umma_tf32_ta(leader, tmem_c, a_hi + 8 * k, b_lo + kPlane + 2 * k,
                                             kDescHi, idesc, 1);
                            }
                        } else {
                            // [main | correction] += hi * [hi | lo], correction += lo * hi
#pragma unroll
                            for (int k = 0; k < kSteps; ++k) {
                                umma_tf32_ta(leader, tmem_d, a_hi + 8 * k, b_lo + 2 * k, kDescHi,
                                             idesc2, (j | k) != 0);
                                umma_tf32_ta(leader, tmem_c, a_lo + 8 * k, b_lo + 2 * k, kDescHi,
                                             idesc, 1);
                            }
                        }
                        umma_commit_if(leader, t_empty_a + 8 * t);
                        b_lo += slot_step;
                        if (++slot == slots) {
                            slot = 0;
                            b_lo = b_first;
                        }
                        if (++t == kT) {
                            t = 0;
                            t_parity ^= 1u;
                        }
                    }
                }
                if (!ok)
                    break;
                umma_commit_if(leader, acc_full_a + 8 * buf);
                buf ^= 1u;
                acc_parity ^= buf ^ 1u;  // flips each time set 0 comes round again
            }
            tile_parity ^= 1u;
        }
        if (!ok)
            give_up(ERR_MMA_WAIT);
        __syncwarp();
    } else if (warp >= 2 + kF32EpilogueWarps) {
        // ---------------- converters: fp32 A tile -> hi and lo planes in tensor memory ----------------
        constexpr int kGroups = f32_groups(BN);
        const int group = (warp - 2 - kF32EpilogueWarps) >> 2;  // takes every kGroups-th stage
        const int q = warp & 3;
        const int row = q * 32 + lane;
        // 16-byte unit u of row r sits at unit u ^ swz of its row
        const int swz = ROWB == 128 ? (row & 7) : ((row >> 1) & 3);
        const int total_iters = my_tiles * (ke - kb);
        // With two groups and an odd number of stages a stage passes from group to group, and a
        // group has not seen the fill before the one it waits for. Where that one is late (its load
        // overtaken by those behind it), its parity is the one that the wait takes for done, and
        // the stage's old tile would be converted. So the wait for the MMAs of step g - kT comes
        // first there: they were issued after every step before them, the fill of step g - stages
        // among those (kT is at most four, and no launch has three stages). With seven stages the
        // group's step before this one has waited for as much.
        const bool passed_on =
                kGroups > 1 && (p.stages & 1) != 0 && p.stages < C::kTStages + kGroups;
        int s = group, t = group;
        uint32_t phase = 0, t_phase = 0;
        // ring slot of the step whose MMAs the next t_empty wait is for (g - kT)
        int s_done = group;
        for (int g = group; g < total_iters; g += kGroups) {
            bool ok = !passed_on || mbar_wait(&t_empty[t], t_phase ^ 1u, abort_flag, p.wait_cycles);
            ok = ok && mbar_wait(&full_bar[s], phase, abort_flag, p.wait_cycles);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                give_up(ERR_PRODUCER_WAIT);
                break;
            }
            const uint4* src = reinterpret_cast<const uint4*>(ring + s * stage_bytes + row * ROWB);
            uint4 v[ROWB / 16];
#pragma unroll
            for (int u = 0; u < ROWB / 16; ++u)
                v[u] = src[u ^ swz];
            ok = mbar_wait(&t_empty[t], t_phase ^ 1u, abort_flag, p.wait_cycles);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                give_up(ERR_PRODUCER_WAIT);
                break;
            }
            if (!p.b_resident && g >= kT) {
                // the MMAs of step g - kT have retired: its ring slot goes back to the producer
                // (on the MMA warp's behalf, whose time is the dearest here)
                if (threadIdx.x % 128 == 64)
                    mbar_arrive(&empty_bar[s_done]);
                s_done += kGroups;
                if (s_done >= p.stages)
                    s_done -= p.stages;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t ta = tmem_base + ((uint32_t)(q * 32) << 16) + kTmemA +
                                (uint32_t)(t * 2 * kChans);
#pragma unroll
            for (int h = 0; h < kChans / 16; ++h) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    split_tf32(v[4 * h + j].x, hi[4 * j + 0], lo[4 * j + 0]);
                    split_tf32(v[4 * h + j].y, hi[4 * j + 1], lo[4 * j + 1]);
                    split_tf32(v[4 * h + j].z, hi[4 * j + 2], lo[4 * j + 2]);
                    split_tf32(v[4 * h + j].w, hi[4 * j + 3], lo[4 * j + 3]);
                }
                tmem_st16(ta + 16 * h, hi);
                tmem_st16(ta + kChans + 16 * h, lo);
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            mbar_arrive(&t_full[t]);
            // The raw tile goes back only now, when its values have been used: a load still on its
            // way to a register is not ordered before the TMA's next write of the slot.
            if (p.b_resident)
                mbar_arrive(&empty_bar[s]);
            s += kGroups;
            if (s >= p.stages) {
                s -= p.stages;
                phase ^= 1u;
            }
            t += kGroups;
            if (t >= kT) {
                t -= kT;
                t_phase ^= 1u;
            }
        }
    } else {
        // ---------------- epilogue: warps 2..9, TMEM lanes 32 * (warp % 4) .. ----------------
        const int q = warp & 3;
        const int row = q * 32 + lane;
        const int half = (warp - 2) >> 2;
        constexpr int kCols = BN / 2;        // columns of this warp
        constexpr int kChunks = kCols / 16;  // ... in 16-column loads
        float* bias_row = reinterpret_cast<float*>(smem + C::kBarBytes) + (warp - 2) * kCols;
        const float4* bias = reinterpret_cast<const float4*>(bias_row);
        // 16- and 32-byte accesses: every row starts on such a boundary when the first does
        const bool vec4 = ((p.ep.dst_pitch | (p.ep.z ? p.ep.z_pitch : 0)) & 3) == 0 &&
                          (((uintptr_t)p.ep.dst | (uintptr_t)p.ep.z) & 15) == 0;
        const bool vec8 = vec4 && (p.ep.dst_pitch & 7) == 0 && ((uintptr_t)p.ep.dst & 31) == 0;
        int local = 0;
        bool ok = true;
        pdl_wait();  // before the first read of z and the first store
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
            const int tile_n = tile % p.n_tiles, tile_m = tile / p.n_tiles;
            const int m = tile_m * kBM + row, n0 = tile_n * BN;
            if (p.n_tiles > 1 || tile == first_tile) {  // once, where one column covers the channels
                __syncwarp();
#pragma unroll
                for (int j = lane; j < kCols; j += 32) {
                    const int ch = n0 + half * kCols + j;
                    bias_row[j] = p.ep.bias && ch < p.oc ? __ldg(p.ep.bias + ch) : 0.f;
                }
                __syncwarp();
            }
            if (p.ep.z && p.splits == 1 && m < p.m_total) {
                const float* zin = p.ep.z + (size_t)m * p.ep.z_pitch + n0 + half * kCols;
#pragma unroll
                for (int j = 0; j < kCols; j += 32)
                    if (n0 + half * kCols + j < p.oc)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(zin + j));
            }
            // running fp32 sums of this thread's accumulators over the tile's segments
            float sum[kCols];
#pragma unroll
            for (int j = 0; j < kCols; ++j)
                sum[j] = 0.f;
            // Adds this warp's columns from `ta` on. (Each load is waited for in the statement that
            // issues it: with a load in flight across other code, a register that it has yet to
            // write must never be spilled, and with this many sums nothing guarantees that.)
            auto add_columns = [&](uint32_t ta) {
#pragma unroll
                for (int c = 0; c < kChunks; ++c) {
                    uint32_t v[16];
                    tmem_ld16(ta + 16 * c, v);
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        sum[16 * c + j] = __fadd_rn(sum[16 * c + j], __uint_as_float(v[j]));
                }
            };
            const uint32_t lane_base =
                    tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * kCols);
            for (int k0 = kb; k0 < ke && ok; k0 += C::kSegIters, ++local) {
                const int buf = local & 1;
                const uint32_t acc_phase = (uint32_t)(local >> 1) & 1u;
                ok = mbar_wait(&acc_full[buf], acc_phase, abort_flag, p.wait_cycles);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) {
                    give_up(ERR_EPILOGUE_WAIT);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if constexpr (C::kWide) {
                    if (k0 + C::kSegIters >= ke) {
                        // last segment: every correction MMA of the tile has retired as well
                        add_columns(lane_base + 2 * BN);
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        mbar_arrive(corr_empty);
                    }
                    add_columns(lane_base + (uint32_t)(buf * BN));
                } else {
                    add_columns(lane_base + (uint32_t)(buf * 2 * BN));
                    add_columns(lane_base + (uint32_t)(buf * 2 * BN + BN));
                }
                // this thread's accumulators are in registers: hand the set back
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                mbar_arrive(&acc_empty[buf]);
            }
            if (!ok)
                break;
            if (p.splits > 1) {
                // (every load of the ring has been consumed and every MMA has retired: the
                // partial tile takes the ring's place)
                float* part = reinterpret_cast<float*>(tiles) + row * C::kPartPitch + half * kCols;
#pragma unroll
                for (int j = 0; j < kCols / 4; ++j)
                    reinterpret_cast<float4*>(part)[j] = make_float4(
                            sum[4 * j], sum[4 * j + 1], sum[4 * j + 2], sum[4 * j + 3]);
            } else if (m < p.m_total && n0 + half * kCols < p.oc) {
                with_act(p.ep.act, [&](auto a) {
                    store_f32_row<kCols, decltype(a)::value>(sum, p.ep, bias, (size_t)m,
                                                             n0 + half * kCols, vec4, vec8);
                });
            }
        }
    }

    if (p.splits > 1) {
        // Every CTA of the cluster comes here, whatever became of its waits. A thread's items lie
        // 256 apart, in one channel quad: bias and residual are fetched while the partial tiles
        // arrive, and the CTA says that it has read the others' before it activates and stores
        // (an arrival behind the stores waits until they have been performed).
        __syncwarp();
        cluster_arrive();
        constexpr int kQuads = BN / 4, kRowStep = 32 * kF32EpilogueWarps / kQuads;
        constexpr int kItems = kBM / 2 / kRowStep;  // at most (two CTAs)
        const int et = (int)threadIdx.x - 64;
        const bool worker = et >= 0 && et < 32 * kF32EpilogueWarps;
        const int rows = kBM / p.splits;
        const int tile_n = first_tile % p.n_tiles, tile_m = first_tile / p.n_tiles;
        const int c = (et & (kQuads - 1)) * 4, ch = tile_n * BN + c;
        const int r0 = rank * rows + et / kQuads;
        const int m0 = tile_m * kBM + r0;
        const int left = min(4, p.oc - ch);
        const bool vec = left == 4 && ((p.ep.dst_pitch | (p.ep.z ? p.ep.z_pitch : 0)) & 3) == 0 &&
                         (((uintptr_t)p.ep.dst | (uintptr_t)p.ep.z) & 15) == 0;
        float bias[4] = {0.f, 0.f, 0.f, 0.f};
        float4 v[kItems], zv[kItems];
        int items = 0;
        if (worker && left > 0) {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j < left && p.ep.bias)
                    bias[j] = __ldg(p.ep.bias + ch + j);
#pragma unroll
            for (int k = 0; k < kItems; ++k) {
                zv[k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (et / kQuads + k * kRowStep < rows && m0 + k * kRowStep < p.m_total) {
                    items = k + 1;
                    if (p.ep.z) {
                        const float* zin = p.ep.z + (size_t)(m0 + k * kRowStep) * p.ep.z_pitch + ch;
                        if (vec) {
                            zv[k] = *reinterpret_cast<const float4*>(zin);
                        } else {
                            zv[k].x = zin[0];
                            zv[k].y = left > 1 ? zin[1] : 0.f;
                            zv[k].z = left > 2 ? zin[2] : 0.f;
                            zv[k].w = left > 3 ? zin[3] : 0.f;
                        }
                    }
                }
            }
        }
        cluster_wait();  // the partial tiles are in place
        if (*abort_flag)
            items = 0;
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            if (k < items) {
                const uint32_t at = smem_u32(tiles) +
                                    (uint32_t)(((r0 + k * kRowStep) * C::kPartPitch + c) * 4);
                // all parts' loads are in flight together (a remote load takes some 250 clocks)
                uint4 x[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (i < p.splits)
                        x[i] = ld_cluster_v4(at, i);
                v[k] = make_float4(__uint_as_float(x[0].x), __uint_as_float(x[0].y),
                                   __uint_as_float(x[0].z), __uint_as_float(x[0].w));
#pragma unroll
                for (int i = 1; i < 8; ++i) {
                    if (i < p.splits) {
                        v[k].x = __fadd_rn(v[k].x, __uint_as_float(x[i].x));
                        v[k].y = __fadd_rn(v[k].y, __uint_as_float(x[i].y));
                        v[k].z = __fadd_rn(v[k].z, __uint_as_float(x[i].z));
                        v[k].w = __fadd_rn(v[k].w, __uint_as_float(x[i].w));
                    }
                }
            }
        }
        __syncwarp();
        cluster_arrive();  // (a release: the loads above are done)
        with_act(p.ep.act, [&](auto a) {
#pragma unroll
            for (int k = 0; k < kItems; ++k) {
                if (k < items) {
                    constexpr int kAct = decltype(a)::value;
                    float4 r;
                    r.x = act_f32<kAct>(v[k].x + bias[0]);
                    r.y = act_f32<kAct>(v[k].y + bias[1]);
                    r.z = act_f32<kAct>(v[k].z + bias[2]);
                    r.w = act_f32<kAct>(v[k].w + bias[3]);
                    if (p.ep.z) {
                        r.x += zv[k].x;
                        r.y += zv[k].y;
                        r.z += zv[k].z;
                        r.w += zv[k].w;
                    }
                    float* out = p.ep.dst + (size_t)(m0 + k * kRowStep) * p.ep.dst_pitch + ch;
                    if (vec) {
                        *reinterpret_cast<float4*>(out) = r;
                    } else {
                        out[0] = r.x;
                        if (left > 1)
                            out[1] = r.y;
                        if (left > 2)
                            out[2] = r.z;
                        if (left > 3)
                            out[3] = r.w;
                    }
                }
            }
        });
        __syncwarp();
        cluster_wait();  // nobody leaves while its partial tile may still be read
    }

    // ---------------- teardown ----------------
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag) {
        if (warp == 1 && lane == 0) {
            umma_commit(drain_bar);
            const long long t0 = clock64();
            while (!mbar_try_wait(drain_bar, 0)) {
                if (clock64() - t0 > p.wait_cycles) {
                    atomicExch(p.status, ERR_DRAIN_WAIT);
                    break;
                }
            }
        }
        for (int i = 0; i < 200; ++i)
            __nanosleep(1000);
        __syncthreads();
    }
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                     "r"(512)
                     : "memory");
    }
}

// ------------------------------------------------------------------------------------------
// general CUDA-core kernel: any shape, groups, odd channel counts; also the small heads
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) conv_f32_direct_kernel(
        ConvF32Args a, const float* __restrict__ src, const float* __restrict__ flt,
        const float* __restrict__ flt_lo, int flt_ic, const float* __restrict__ bias,
        const float* z, float* dst) {
    pdl_start();
    // flt: the K-major filter [OC][KH][KW][flt_ic], or its hi plane with the lo plane beside it
    const size_t total = (size_t)a.m * a.oc;
    const int icpg = a.ic / a.groups, ocpg = a.oc / a.groups;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int o = (int)(idx % a.oc);
        const size_t m = idx / a.oc;
        const int ox = (int)(m % a.ow);
        const size_t t = m / a.ow;
        const int oy = (int)(t % a.oh);
        const int n = (int)(t / a.oh);
        const int g = o / ocpg;
        const size_t w0 = (size_t)o * a.kh * a.kw * flt_ic;
        float acc = 0.f;
        for (int fy = 0; fy < a.kh; ++fy) {
            const int iy = oy * a.sh + fy - a.ph;
            if ((unsigned)iy >= (unsigned)a.ih)
                continue;
            for (int fx = 0; fx < a.kw; ++fx) {
                const int ix = ox * a.sw + fx - a.pw;
                if ((unsigned)ix >= (unsigned)a.iw)
                    continue;
                const float* s = src + (((size_t)n * a.ih + iy) * a.iw + ix) * a.src_pitch +
                                 g * icpg;
                const float* wk = flt + w0 + (size_t)(fy * a.kw + fx) * flt_ic;
                if (flt_lo) {
                    const float* wl = flt_lo + (wk - flt);
                    for (int c = 0; c < icpg; ++c)
                        acc = fmaf(s[c], __fadd_rn(wk[c], wl[c]), acc);
                } else {
                    for (int c = 0; c < icpg; ++c)
                        acc = fmaf(s[c], wk[c], acc);
                }
            }
        }
        float r = acc + (bias ? bias[o] : 0.f);
        with_act(a.act, [&](auto k) { r = act_f32<decltype(k)::value>(r); });
        if (z)
            r += z[m * a.z_pitch + o];
        dst[m * a.dst_pitch + o] = r;
    }
}

// OIHW / [G][OCpg][ICpg][KH][KW] fp32 -> [OC][KH][KW][ICpg]
__global__ void __launch_bounds__(256) pack_filter_f32_plain_kernel(
        const float* __restrict__ src, float* __restrict__ dst, int oc, int icpg, int kh, int kw) {
    const size_t total = (size_t)oc * icpg * kh * kw;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
         i += (size_t)gridDim.x * blockDim.x) {
        const int c = (int)(i % icpg);
        size_t t = i / icpg;
        const int fx = (int)(t % kw);
        t /= kw;
        const int fy = (int)(t % kh);
        const int o = (int)(t / kh);
        dst[i] = src[(((size_t)o * icpg + c) * kh + fy) * kw + fx];
    }
}

// [rows][k] -> [rows][4 k4], zeros behind the k values. Bound by HBM: 8 bytes per element.
__global__ void __launch_bounds__(256) pad_rows_f32_kernel(
        const float* __restrict__ src, float4* __restrict__ dst, long long rows, int k, int k4) {
    pdl_start();
    const long long total = rows * k4;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / k4;
        const int c = (int)(i - r * k4) * 4;
        const float* s = src + r * k + c;
        dst[i] = make_float4(s[0], c + 1 < k ? s[1] : 0.f, c + 2 < k ? s[2] : 0.f, c + 3 < k ? s[3] : 0.f);
    }
}

int grid_1d(size_t work, int block) {
    size_t g = (work + block - 1) / block;
    const size_t most = (size_t)sm_count() * 16;
    if (g > most)
        g = most;
    return g < 1 ? 1 : (int)g;
}

template <int BN, int ROWB>
bool f32_kernel_ready() {
    static KernelReady ready;
    return ready.smem(conv_f32_umma_kernel<BN, ROWB>, F32Cfg<BN, ROWB>::kDynamic);
}

template <int BN, int ROWB>
int f32_clusters(int size) {
    static ClusterCapacity capacity;
    if (!f32_kernel_ready<BN, ROWB>())
        return 0;
    return capacity.clusters(conv_f32_umma_kernel<BN, ROWB>, size, f32_threads(BN),
                             F32Cfg<BN, ROWB>::kDynamic);
}

template <int BN, int ROWB>
int launch_f32_kernel(
        const CUtensorMap& ma, const CUtensorMap& mb, F32ConvParams& p, cudaStream_t st) {
    using C = F32Cfg<BN, ROWB>;
    if (!f32_kernel_ready<BN, ROWB>())
        return check_launch("conv_f32_umma smem attribute");
    // The filter stays resident where one tile column covers the channels and enough A stages
    // fit behind it (a TMA round trip is four to five stages of conversion).
    constexpr int kResidentStages = 5;
    const long long b_all = (long long)p.k_iters * C::kBBytes;
    p.b_resident = p.splits == 1 && p.n_tiles == 1 && p.m_tiles > sm_count() &&
                   b_all + kResidentStages * C::kABytes <= C::kTileBudget;
    const int stage = C::kABytes + (p.b_resident ? 0 : C::kBBytes);
    int stages = (int)((C::kTileBudget - (p.b_resident ? b_all : 0)) / stage);
    p.stages = stages > kMaxStages ? kMaxStages : stages;
    const int total = p.m_tiles * p.n_tiles;
    int grid = total * p.splits;
    if (p.splits == 1 && grid > sm_count())
        grid = sm_count();
    if (tuning().debug)
        fprintf(stderr, "conv_f32_umma<%d,%d>: grid %d tiles %d k_iters %d stages %d resident %d "
                "splits %d\n", BN, ROWB, grid, total, p.k_iters, p.stages, p.b_resident, p.splits);
    launch_pdl_cluster(Writes{p.ep.dst, (size_t)p.m_total * p.ep.dst_pitch * 4}, conv_f32_umma_kernel<BN, ROWB>, dim3(grid), dim3(f32_threads(BN)),
                       (size_t)C::kDynamic, p.splits, st, ma, mb, p);
    return check_launch("conv_f32_umma");
}

int f32_cluster_capacity(int bn, int rowb, int size) {
    if (rowb == 128)
        return bn == 32   ? f32_clusters<32, 128>(size)
               : bn == 64 ? f32_clusters<64, 128>(size)
                          : f32_clusters<128, 128>(size);
    return bn == 32   ? f32_clusters<32, 64>(size)
           : bn == 64 ? f32_clusters<64, 64>(size)
                      : f32_clusters<128, 64>(size);
}

// Tile width and K split for a problem of `m_tiles` x `oc` with `k_iters` steps of `rowb` bytes:
// the pair with the shortest estimated time of its busiest SM. Clocks per step and tile: 12
// MMAs of 64 clocks for 128 columns, half that for 64, and for 32 what the handshakes of a step
// cost. A tile that is its CTA's only one has nothing to hide its end behind: wide tiles cost
// more there (128 -> 128 1x1 over 52 x 52: 4.6 us with 32 columns, 5.3 with 64, 7.8 with 128). A
// split adds the exchange of the partial tiles; it is taken only where the clusters all run at
// once. (512 -> 128 1x1 over 26 x 26: 5.8 us as 24 tiles split in four, 6.8 as 12 in eight.) Over 160
// layers that are in no network here (16 to 512 channels to 16 to 512, 25 to 20000 pixels) the choice is 2 %
// on average behind the best of all widths and splits; one layer (16 -> 85 3x3 over 2 x 13 x 13, unsplit 6.9 us,
// split 4.5) is 52 % off, all others at most 15 %.
struct F32Choice {
    int bn, splits;
    bool half;  // 128 columns, from fp16 planes
};
int f32_step_clocks(int bn, int rowb) { return (bn == 128 ? 850 : bn == 64 ? 500 : 420) * rowb / 128; }
int f32_end_clocks(int bn) { return bn == 128 ? 2500 : bn == 64 ? 1500 : 1000; }  // sums, activation, stores
F32Choice choose_f32_tile(const ConvF32Args& a, bool planes) {
    const int rowb = a.ic <= 16 ? 64 : 128, oc = a.oc;
    const int m_tiles = (a.m + kBM - 1) / kBM;
    const int k_iters = a.kh * a.kw * (conv_f32_padded_ic(a.ic) * 4 / rowb);
    F32Choice c{128, 1, false};
    const int sms = sm_count();
    long long best = -1;
    for (int b = 128; b >= 32; b /= 2) {
        if (b > 32 && oc <= b / 2)
            continue;
        const int step = f32_step_clocks(b, rowb), tile_end = f32_end_clocks(b);
        const long long tiles = (long long)m_tiles * ((oc + b - 1) / b);
        for (int s = 1; s <= 8; s *= 2) {
            if (s > 1 && (k_iters / s < 2 || tiles > sms / s || tiles > f32_cluster_capacity(b, rowb, s)))
                break;
            const long long waves = s > 1 ? 1 : (tiles + sms - 1) / sms;
            const int alone = waves > 1 ? 0 : b == 128 ? 3000 : b == 64 ? 900 : 0;
            const long long clocks =
                    waves * ((long long)((k_iters + s - 1) / s) * step + tile_end + alone) +
                    (s > 1 ? 2500 : 0);
            if (best < 0 || clocks < best) {
                best = clocks;
                c.bn = b;
                c.splits = s;
            }
        }
    }
    // 128 columns from fp16 planes (conv_f32_half.cu): two rows of A in the time of 1.64 here (32 x 80 x 80
    // pixels, 128 -> 128 3x3: 282 us and 224; 32 x 20 x 20, 256 -> 256: 100 as 64 columns, 72)
    const long long waves = ((long long)m_tiles * ((oc + 127) / 128) + sms - 1) / sms;
    const bool fits = planes && waves <= kExactTiles;
    c.half = fits && waves * ((long long)((k_iters + 1) / 2) * 1395 + 2500 + (waves > 1 ? 0 : 3000)) < best;
    if (tuning().f32_bn == 32 || tuning().f32_bn == 64 || tuning().f32_bn == 128)
        c.bn = tuning().f32_bn;
    if (tuning().f32_split == 1 || tuning().f32_split == 2 || tuning().f32_split == 4 ||
        tuning().f32_split == 8)
        c.splits = k_iters >= tuning().f32_split ? tuning().f32_split : 1;
    if (tuning().f32_bn || tuning().f32_split || tuning().f32_half != 1)
        c.half = fits && tuning().f32_half == 2;
    return c;
}

bool plain_matrix(const ConvF32Args& a) {
    return a.kh == 1 && a.kw == 1 && a.sh == 1 && a.sw == 1 && a.ph == 0 && a.pw == 0;
}

}  // namespace

// channels the packed (split) filter holds per tap: ic rounded up to a whole TMA row
int conv_f32_padded_ic(int ic) {
    return ic <= 16 ? 16 : (ic + 31) / 32 * 32;
}

// the clocks of one tile among others, by the estimates of choose_f32_tile
long long conv_f32_tile_clocks(const ConvF32Args& a, int bn) {
    const int rowb = a.ic <= 16 ? 64 : 128;
    return (long long)a.kh * a.kw * (conv_f32_padded_ic(a.ic) * 4 / rowb) * f32_step_clocks(bn, rowb) +
           f32_end_clocks(bn);
}

size_t conv_f32_split_filter_floats(const ConvF32Args& a) {
    return 2 * (size_t)a.oc * a.kh * a.kw * conv_f32_padded_ic(a.ic) +
           (conv_f32_half_planes(a) ? conv_f32_half_filter_floats(a) : 0) +
           (conv_f32_patch_planes(a) ? conv_f32_patch_filter_floats(a) : 0);
}

// What a packed filter holds follows from the filter's own groups, channels and extent and from nothing else:
// a filter packed under one input, stride and padding may be used under another, and so may the second
// operand of a matrix product as a 1x1 filter.
//
// The two planes: channel counts the tensor-core kernel takes, rows the TMA can address (16-byte multiples).
// A last, partial row of 32 channels is filled with zeros by the load; the im2col form asks
// for whole rows of a tensor at least that wide.
bool conv_f32_split_planes(const ConvF32Args& a) {
    if (a.groups != 1 || a.ic % 4 != 0)
        return false;
    return (a.kh == 1 && a.kw == 1) || a.ic == 16 || a.ic >= 32;
}
const float* conv_f32_channel_words(const ConvF32Args& a, const float* flt_packed) {
    const size_t plane = (size_t)a.oc * a.kh * a.kw * conv_f32_padded_ic(a.ic);
    if (conv_f32_half_planes(a))
        return flt_packed + 3 * plane;
    return conv_f32_patch_planes(a) ? flt_packed + 2 * plane + conv_f32_patch_words_at(a) : nullptr;
}
// Filters that 128-channel tiles can be taken for (rows of 128 bytes, more than 64 channels) hold the fp16
// planes as well: which kernel runs is known only with the batch.
bool conv_f32_half_planes(const ConvF32Args& a) {
    return (a.forms & F32_HALF_PLANES) && conv_f32_split_planes(a) && a.ic > 16 && a.oc > 64;
}

// Images of `src` the activation's im2col map describes (see descriptor_images in internal.h)
static int f32_descriptor_images(const ConvF32Args& a, const float* src) {
    constexpr size_t kMinMapBytes = 131072;
    const size_t image = (size_t)a.ih * a.iw * a.src_pitch * 4;
    if ((size_t)a.n * image >= kMinMapBytes)
        return a.n;
    const size_t images = (kMinMapBytes + image - 1) / image;
    return readable_through(src, images * image) ? (int)images : 0;
}

// Tensor-core path: dense, an eligible channel count, 16-byte aligned operands and pitches,
// and, with a spatial filter, 128 KiB of readable memory behind `src` for the TMA map.
bool conv_f32_umma_supported(const ConvF32Args& a, const float* src, const float* dst) {
    if (!conv_f32_split_planes(a) || !(plain_matrix(a) || a.ic == 16 || a.ic >= 32))
        return false;
    if (a.kh * a.kw > 49 || a.ph > 64 || a.pw > 64 || a.sh > 8 || a.sw > 8)
        return false;
    if ((size_t)a.n * a.ih * a.iw >= (1ull << 31) || (size_t)a.m >= (1ull << 31))
        return false;
    if (((uintptr_t)src | (uintptr_t)dst) & 15)
        return false;
    if (a.src_pitch & 3)
        return false;
    return plain_matrix(a) || f32_descriptor_images(a, src) != 0;
}

int launch_conv_f32_pack_filter_split(
        const ConvF32Args& a, const float* flt_oihw, float* out, cudaStream_t st) {
    const int icp = conv_f32_padded_ic(a.ic);
    const size_t plane = (size_t)a.oc * a.kh * a.kw * icp;
    pack_filter_f32_kernel<<<grid_1d(plane, 256), 256, 0, st>>>(flt_oihw, out, a.oc, a.ic, icp,
                                                                 a.kh, a.kw);
    int rc = check_launch("pack_filter_f32");
    out += 2 * plane;
    if (!rc && conv_f32_half_planes(a)) {
        rc = launch_conv_f32_pack_filter_half(a, flt_oihw, out, st);
        out += conv_f32_half_filter_floats(a);
    }
    return rc || !conv_f32_patch_planes(a) ? rc : launch_conv_f32_pack_filter_patch(a, flt_oihw, out, st);
}

int launch_conv_f32_pack_filter_plain(
        const ConvF32Args& a, const float* flt_oihw, float* out, cudaStream_t st) {
    const int icpg = a.ic / a.groups;
    const size_t total = (size_t)a.oc * icpg * a.kh * a.kw;
    pack_filter_f32_plain_kernel<<<grid_1d(total, 256), 256, 0, st>>>(flt_oihw, out, a.oc, icpg,
                                                                       a.kh, a.kw);
    return check_launch("pack_filter_f32_plain");
}

int launch_matmul_f32_pack_split(
        int k, int n, const float* b, float* out, cudaStream_t st) {
    const int kp = conv_f32_padded_ic(k);
    dim3 grid((n + 31) / 32, (kp + 31) / 32), block(32, 8);
    if (grid.y > 65535)
        return set_error(ST_OUT_OF_RANGE, "matmul: k = %d exceeds the grid limit", k);
    pack_matrix_f32_kernel<<<grid, block, 0, st>>>(b, out, k, n, kp);
    return check_launch("pack_matrix_f32");
}

int launch_matmul_f32_pack_b(const ConvF32Args& a, const float* b, float* out, cudaStream_t st) {
    const int rc = launch_matmul_f32_pack_split(a.ic, a.oc, b, out, st);
    out += 2 * (size_t)a.oc * conv_f32_padded_ic(a.ic);
    return rc || !conv_f32_half_planes(a) ? rc : launch_matmul_f32_pack_half(a.ic, a.oc, b, out, st);
}

int launch_conv_f32_direct(
        const ConvF32Args& a, const float* src, const float* flt_packed, const float* bias,
        const float* z, float* dst, cudaStream_t st) {
    const bool split = conv_f32_split_planes(a);
    const int icp = split ? conv_f32_padded_ic(a.ic) : a.ic / a.groups;
    const float* lo = split ? flt_packed + (size_t)a.oc * a.kh * a.kw * icp : nullptr;
    launch_pdl(Writes{dst, (size_t)a.m * a.dst_pitch * 4}, conv_f32_direct_kernel, dim3(grid_1d((size_t)a.m * a.oc, 256)), dim3(256), 0, st, a,
               src, flt_packed, lo, icp, bias, z, dst);
    return check_launch("conv_f32_direct");
}

// `planes`: the fp16 planes of the filter, where the choice may fall on them. `raw`: the second operand of a
// matrix product, of which these planes alone were made then, or null
static int launch_f32_tensor(
        const ConvF32Args& a, const float* src, const float* flt_split, const float* planes, const float* raw,
        const F32Choice& choice, const float* bias, const float* z, float* dst, cudaStream_t st) {
    const DriverApi& api = driver_api();
    if (!api.ok)
        return set_error(ST_RUNTIME, "cuTensorMapEncode* entry points not found in the driver");
    if ((uintptr_t)flt_split & 15)
        return set_error(ST_INVALID_LAYOUT, "the filter must be 16-byte aligned");

    const int rowb = a.ic <= 16 ? 64 : 128;
    const int chans = rowb / 4;
    const int icp = conv_f32_padded_ic(a.ic);
    const CUtensorMapSwizzle swz =
            rowb == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B;
    const int taps = a.kh * a.kw;
    const bool a_tiled = plain_matrix(a);
    F32ConvParams p;
    p.m_tiles = (a.m + kBM - 1) / kBM;
    p.cblocks = icp / chans;
    p.k_iters = taps * p.cblocks;
    const int bn = choice.bn;
    p.splits = choice.splits;
    CUtensorMap map_a, map_b;
    if (a_tiled) {
        cuuint64_t dims[2] = {(cuuint64_t)a.ic, (cuuint64_t)a.m};
        cuuint64_t strides[1] = {(cuuint64_t)a.src_pitch * 4};
        cuuint32_t box[2] = {(cuuint32_t)chans, (cuuint32_t)kBM};
        cuuint32_t estr[2] = {1, 1};
        CUresult r = api.tiled(&map_a, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)src, dims, strides,
                               box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            return set_error(ST_RUNTIME, "cuTensorMapEncodeTiled(f32 activation) failed: %d", (int)r);
    } else {
        const int images = f32_descriptor_images(a, src);
        if (images == 0)
            return set_error(ST_INVALID_LAYOUT, "activation below 128 KiB outside a registered range");
        cuuint64_t dims[4] = {(cuuint64_t)a.ic, (cuuint64_t)a.iw, (cuuint64_t)a.ih,
                              (cuuint64_t)images};
        cuuint64_t strides[3] = {(cuuint64_t)a.src_pitch * 4, (cuuint64_t)a.iw * a.src_pitch * 4,
                                 (cuuint64_t)a.ih * a.iw * a.src_pitch * 4};
        int lower[2] = {-a.pw, -a.ph};
        int upper[2] = {(a.ow - 1) * a.sw - a.pw - (a.iw - 1), (a.oh - 1) * a.sh - a.ph - (a.ih - 1)};
        cuuint32_t estr[4] = {1, (cuuint32_t)a.sw, (cuuint32_t)a.sh, 1};
        CUresult r = api.im2col(&map_a, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (void*)src, dims, strides,
                                lower, upper, chans, kBM, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                                CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            return set_error(ST_RUNTIME, "cuTensorMapEncodeIm2col(f32) failed: %d", (int)r);
    }
    if (choice.half)
        return launch_conv_f32_half(a, map_a, a_tiled, src, planes, raw ? raw : flt_split, raw != nullptr, bias, z,
                                    dst, st);
    {
        const cuuint64_t k_total = (cuuint64_t)taps * icp;
        cuuint64_t dims[2] = {k_total, (cuuint64_t)2 * a.oc};
        cuuint64_t strides[1] = {k_total * 4};
        cuuint32_t box[2] = {(cuuint32_t)chans, (cuuint32_t)bn};
        cuuint32_t estr[2] = {1, 1};
        CUresult r = api.tiled(&map_b, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)flt_split, dims,
                               strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            return set_error(ST_RUNTIME, "cuTensorMapEncodeTiled(f32 filter) failed: %d", (int)r);
    }
    p.m_total = a.m;
    p.oc = a.oc;
    p.oh = a.oh;
    p.ow = a.ow;
    p.taps_w = a.kw;
    p.sh = a.sh;
    p.sw = a.sw;
    p.base_h = -a.ph;
    p.base_w = -a.pw;
    p.n_tiles = (a.oc + bn - 1) / bn;
    p.a_tiled = a_tiled ? 1 : 0;
    p.b_lo_offset = a.oc;
    p.ep.oc = a.oc;
    p.ep.act = a.act;
    p.ep.bias = bias;
    p.ep.z = z;
    p.ep.z_pitch = a.z_pitch;
    p.ep.dst = dst;
    p.ep.dst_pitch = a.dst_pitch;
    p.status = device_status_word(st);
    if (!p.status)
        return ST_MALLOC;
    p.wait_cycles = kWaitCycles;
    if (rowb == 128)
        return bn == 32   ? launch_f32_kernel<32, 128>(map_a, map_b, p, st)
               : bn == 64 ? launch_f32_kernel<64, 128>(map_a, map_b, p, st)
                          : launch_f32_kernel<128, 128>(map_a, map_b, p, st);
    return bn == 32   ? launch_f32_kernel<32, 64>(map_a, map_b, p, st)
           : bn == 64 ? launch_f32_kernel<64, 64>(map_a, map_b, p, st)
                      : launch_f32_kernel<128, 64>(map_a, map_b, p, st);
}

static bool takes_patches(const ConvF32Args& a) {
    return conv_f32_patch_shape(a) && !tuning().f32_bn && !tuning().f32_split && conv_f32_patch_pays(a);
}

int conv_f32_forms(const ConvF32Args& a) {
    if (!conv_f32_split_planes(a))
        return 0;
    return takes_patches(a) ? F32_PATCH_PLANES
                            : choose_f32_tile(a, conv_f32_half_planes(a)).half ? F32_HALF_PLANES : 0;
}

int launch_conv_f32_umma(
        const ConvF32Args& a, const float* src, const float* flt_split, const float* bias,
        const float* z, float* dst, cudaStream_t st) {
    // (a residual in the result's own place: the kernels on fp16 planes may store a tile twice)
    const bool fp16_planes = !a.tf32_only && z != dst;
    const bool has = conv_f32_half_planes(a);
    const float* planes = flt_split + 2 * (size_t)a.oc * a.kh * a.kw * conv_f32_padded_ic(a.ic);
    if (fp16_planes && takes_patches(a) && ((uintptr_t)flt_split & 15) == 0)
        return launch_conv_f32_patch(a, src, planes + (has ? conv_f32_half_filter_floats(a) : 0), flt_split, bias,
                                     z, dst, st);
    return launch_f32_tensor(a, src, flt_split, planes, nullptr, choose_f32_tile(a, has && fp16_planes), bias,
                             z, dst, st);
}

// ---- a matrix product with both operands as the caller has them ----
static bool product_pads(int k, const float* a) {
    return k % 4 != 0 || ((uintptr_t)a & 15) != 0;
}

size_t matmul_f32_scratch_floats(const ConvF32Args& a, const float* src) {
    const int kp = conv_f32_padded_ic(a.ic);
    const size_t b = 2 * (size_t)a.oc * kp + (size_t)(a.oc + 3) / 4 * 4;
    return b + (product_pads(a.ic, src) ? (size_t)a.m * ((a.ic + 3) / 4 * 4) : 0);
}

// Which planes of B are made is decided with the sizes of the product. Rows of A that the TMA cannot
// address are copied to a pitch that it can: a 230 x 617 x 1974 product takes 22.5 us, 556 on the CUDA cores.
int launch_matmul_f32(
        ConvF32Args a, const float* src, const float* b, float* c, float* scratch, cudaStream_t st) {
    const F32Choice choice = choose_f32_tile(a, a.ic > 16 && a.oc > 64);
    const int kp = conv_f32_padded_ic(a.ic);
    float* packed = scratch;
    if (product_pads(a.ic, src)) {
        float* rows = scratch + 2 * (size_t)a.oc * kp + (size_t)(a.oc + 3) / 4 * 4;
        a.src_pitch = (a.ic + 3) / 4 * 4;
        const size_t total = (size_t)a.m * a.src_pitch;
        launch_pdl(Writes{rows, total * 4}, pad_rows_f32_kernel, dim3(grid_1d(total / 4, 256)), dim3(256), 0,
                   st, src, reinterpret_cast<float4*>(rows), (long long)a.m, a.ic, (int)a.src_pitch / 4);
        const int rc = check_launch("pad_rows_f32");
        if (rc)
            return rc;
        src = rows;
    }
    const int rc = choice.half ? launch_matmul_f32_pack_half(a.ic, a.oc, b, packed, st)
                               : launch_matmul_f32_pack_split(a.ic, a.oc, b, packed, st);
    return rc ? rc : launch_f32_tensor(a, src, packed, packed, b, choice, nullptr, nullptr, c, st);
}

}  // namespace mb200
