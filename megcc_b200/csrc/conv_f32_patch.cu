// fp32 ConvBias 3x3, stride 1, padding 1, on the sm_100a tensor cores with halo-patch input tiles.
//
// With im2col loads (conv_f32.cu, conv_f32_half.cu) every pixel is fetched, and split into its planes, once per
// filter tap: the TMA takes four clocks for each of its rows, and the converters' chain is the longest of the
// kernel. Here an output tile is a patch of 16 x 8 pixels; its 18 x 10 input pixels are fetched and split
// ONCE per 64 channels, into two fp16 planes in shared memory, [pixel][64 channels] with the 128-byte
// swizzle. Every tap is those planes addressed from its own pixel (the swizzle is a function of the
// shared-memory address, so a shifted start needs nothing else), rows of eight pixels, 10 pixels apart.
//
// Arithmetic as in conv_f32_half.cu: each pixel's 64 channels share a power of two, a channel's filter another;
// 2^-12 (lo*hi + hi*lo) + hi*hi, a segment (one tap x 64 channels) in accumulators of its own, whose sum is taken
// into fp32 registers times the pixel's factor, which is the tap's pixel here. Tiles whose operands lie too far
// apart for that are put off and taken from tf32 planes at the kernel's end (conv_f32_exact.cuh).
//
// What bounds it: the MMAs' operands from shared memory (A 4 KB, B 1 to 4 KB each, 128 bytes a clock: 40, 48,
// 64 clocks for 32, 64, 128 columns; issued one in 60 to 75) and whatever else takes that memory's time;
// with 128 columns also the hand-over of every segment's sums to the epilogue (480 clocks). Hence the filter
// is packed as it lies in shared memory and comes in one contiguous copy per group of taps (boxes of a
// tensor map took 5.7 clocks a row: 32 x 320 x 320, 16 -> 32, 600 us, then 430), stays there where it is the only
// one, pixels go from global memory to the planes by way of registers, a block ahead, and results leave turned
// round. 32 images, us, im2col tiles and here: 80 x 80, 64 -> 64: 88, 61; 128 -> 128: 224, 184; 160 x 160, 32 -> 32:
// 164, 123; 320 x 320, 16 -> 32: 419, 388.
//
// Structure: persistent CTAs, warp 0 filter producer, warp 1 MMA issuer and TMEM owner, warps 2..9 epilogue,
// warps 10..17 converters (fp32 patch -> planes), bounded waits.
//
// Replaces, for the fp32 configurations, the reference's im2col + 4x12 SIMD GEMM
// (compiler/lib/KernelGen/GeneralIntrinsic/ConvKernel/Fp32Im2col.cpp:122-217).
#include <stdio.h>

#include "conv_f32_epilogue.cuh"
#include "conv_f32_exact.cuh"
#include "conv_f32_split.cuh"
#include "f32_internal.h"
#include "pdl.h"
#include "tuning.h"
#include "umma_ptx.cuh"

namespace mb200 {

using namespace umma;

namespace {

constexpr int kBM = 128;
constexpr int kTH = 16, kTW = 8;          // output patch; a row of eight pixels is a core-matrix group
constexpr int kPH = kTH + 2, kPW = kTW + 2;
constexpr int kPixels = kPH * kPW;
constexpr int kTaps = 9;
constexpr int kBlock = 64;                // channels split at a time
constexpr int kPlane = 23 * 1024;         // 180 pixels x 128 bytes, up to the swizzle's 1024
constexpr int kConverterWarps = 8;
static_assert(kPixels * 128 <= kPlane, "a plane");

template <int BN>
struct Cfg {
    // taps per hand-over between producer, MMAs and epilogue: with few columns a barrier costs as much as a
    // tap's MMAs
    static constexpr int kGroup = BN == 128 ? 1 : 3;
    static constexpr int kTapBytes = 2 * BN * kBlock * 2;  // both planes of a tap's filter
    static constexpr int kBBytes = kGroup * kTapBytes;
    // groups in flight, each with accumulators of its own: the MMAs go on while the epilogue stores a tile
    static constexpr int kBars = BN == 64 ? 2 : 4;
    // (32 columns: a whole block's filter, which then stays where it is the only one)
    static constexpr int kBStages = BN == 64 ? 2 : 3;
    static constexpr int kEpilogueWarps = 8;
    static constexpr int kCols = BN / (kEpilogueWarps / 4);    // accumulator columns of a warp
    static constexpr int kTurn = kCols < 32 ? kCols : 32;      // ... turned round at a time
    static constexpr int kTurnBytes = 32 * kTurn * 4;
    static constexpr int kThreads = 64 + 32 * (kEpilogueWarps + kConverterWarps);
    static constexpr int kLateOff = 240;  // LateTiles
    static constexpr int kFactorOff = (kLateOff + (int)sizeof(LateTiles) + 15) / 16 * 16;
    // Pixel factors: the converters write those of block n + 2 when the MMAs of block n have retired, and the
    // epilogue is at most kBars groups behind these.
    static constexpr int kFactorSets = kBars * kGroup < kTaps ? 3 : 4;
    // Two sets of a tile column's factors and biases. (A warp is never two tiles ahead of another.)
    static constexpr int kChannelOff = kFactorOff + (kFactorSets * kPixels * 4 + 15) / 16 * 16;
    static constexpr int kFront = kChannelOff + 2 * 2 * BN * 4;
    static constexpr int kFrontBytes = (kFront + 1023) / 1024 * 1024;
    static constexpr int kPlaneBytes = 2 * 2 * kPlane;  // two buffers of two planes
    static constexpr int kTotal =
            kFrontBytes + kPlaneBytes + kBStages * kBBytes + kEpilogueWarps * kTurnBytes;
    static constexpr int kDynamic = kTotal + 1024;
    static_assert(kBStages <= kBars, "a segment's barrier is reused behind its filter's stage");
    static_assert(kBars * kGroup * BN <= 512, "tensor memory");
    static_assert(kDynamic <= 227 * 1024, "shared memory");
    static_assert(kBars * kGroup < 2 * kTaps, "factor sets");
    static_assert((64 + BN / 2) * 1024 <= kPlaneBytes + kBStages * kBBytes, "a tile from tf32 planes");
};

// A tile's rows for the general form: patch rows of eight pixels
struct PatchPixel {
    int img, y0, x0, oh, ow;
    __device__ __forceinline__ ExactPixel operator()(int row) const {
        const int y = y0 + (row >> 3), x = x0 + (row & 7);
        return ExactPixel{img, y, x, y < oh && x < ow};
    }
};

struct PatchF32Params {
    int n, oh, ow, oc, ic;
    const float* src;
    long long src_pitch;
    int blocks;              // of 64 input channels
    int tiles_y, tiles_x, m_tiles, n_tiles;
    F32Epilogue ep;
    const uint8_t* filter;   // [tile column][block][tap][plane][BN][64 channels], rows swizzled as in shared memory
    const float* factor;     // per output channel: what a unit of the accumulated sums stands for (channel_word)
    ExactOperands exact;
    int* status;
    __device__ __forceinline__ PatchPixel pixel(int tile) const {
        const int m = tile / n_tiles, per_image = tiles_y * tiles_x, img = m / per_image, r = m - img * per_image;
        return PatchPixel{img, r / tiles_x * kTH, r % tiles_x * kTW, oh, ow};
    }
};

// both operands in shared memory (descriptors as their two words); issued by the lane whose `leader` is
// non-zero. SHIFT: what is in the accumulator counts 2^-SHIFT times
template <int SHIFT = 0>
__device__ __forceinline__ void umma_f16_ss(
        uint32_t leader, uint32_t tmem_d, uint32_t a_lo, uint32_t b_lo, uint32_t a_hi, uint32_t b_hi,
        uint32_t idesc, uint32_t accumulate) {
    asm volatile(
            "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
            "mov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
            "setp.ne.b32 p, %6, 0;\n\tsetp.ne.b32 q, %7, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %5, p, %8;\n\t}" ::"r"(tmem_d),
            "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(leader), "n"(SHIFT)
            : "memory");
}

// contiguous bytes, addresses and size multiples of 16
__device__ __forceinline__ void bulk_load_if(
        uint32_t leader, uint32_t smem, const void* from, uint32_t bytes, uint32_t bar) {
    asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t"
            "@q cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n\t}" ::"r"(
                    smem),
            "l"(from), "r"(bytes), "r"(bar), "r"(leader)
            : "memory");
}

// three times 16 columns, loads and wait in one statement
__device__ __forceinline__ void tmem_ld16x3(uint32_t a, uint32_t b, uint32_t c, uint32_t (&v)[48]) {
    asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%48];\n\t"
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%49];\n\t"
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47}, [%50];\n\t"
            "tcgen05.wait::ld.sync.aligned;"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
              "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
              "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
              "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
              "=r"(v[31]), "=r"(v[32]), "=r"(v[33]), "=r"(v[34]), "=r"(v[35]), "=r"(v[36]),
              "=r"(v[37]), "=r"(v[38]), "=r"(v[39]), "=r"(v[40]), "=r"(v[41]), "=r"(v[42]),
              "=r"(v[43]), "=r"(v[44]), "=r"(v[45]), "=r"(v[46]), "=r"(v[47])
            : "r"(a), "r"(b), "r"(c)
            : "memory");
}

template <int N>
struct Number {
    static constexpr int value = N;
};

// a CTA's tile: channel column fastest, then along the image
struct TilePos {
    int n0, img, y0, x0;
    __device__ __forceinline__ TilePos(int tile, int bn, const PatchF32Params& p) {
        const int m = tile / p.n_tiles;
        n0 = (tile - m * p.n_tiles) * bn;
        const int per_image = p.tiles_y * p.tiles_x;
        img = m / per_image;
        const int r = m - img * per_image, ty = r / p.tiles_x;
        y0 = ty * kTH;
        x0 = (r - ty * p.tiles_x) * kTW;
    }
};

// A warp's rows: four of the patch, eight pixels each (a lane's own first row lies in the first of them)
struct PatchRows {
    const PatchF32Params& p;
    size_t first;
    int y0, x0;
    __device__ __forceinline__ bool there(int row0, int row) const {
        return y0 + (row >> 3) < p.oh && x0 + row0 + (row & 7) < p.ow;
    }
    __device__ __forceinline__ int step(int row) const { return (row >> 3) * p.ow + (row & 7); }
};

// OIHW fp32 -> the filter's planes and channel words, a block per channel of the (padded) tile columns
__global__ void __launch_bounds__(256) pack_filter_patch_kernel(
        const float* __restrict__ src, uint8_t* __restrict__ out, uint32_t* __restrict__ word, int oc, int ic,
        int blocks, int bn) {
    __shared__ Magnitudes shared[8];
    const int o = blockIdx.x, column = o / bn, row = o - column * bn;
    const float* w = src + (size_t)o * ic * kTaps;
    const int count = o < oc ? ic * kTaps : 0;
    Magnitudes of = Magnitudes::none();
    for (int i = threadIdx.x; i < count; i += 256)
        of.take(w[i]);
    of = block_magnitudes(of, shared);
    const uint32_t field = scale_field(of.largest);
    if (threadIdx.x == 0)
        word[o] = of.word();
    const size_t plane = (size_t)bn * kBlock * 2;
    for (int i = threadIdx.x; i < blocks * kTaps * kBlock; i += 256) {
        const int segment = i / kBlock, k = i - segment * kBlock;
        const int block = segment / kTaps, tap = segment - block * kTaps, c = block * kBlock + k;
        uint32_t h, l;
        split_f16(c < ic && o < oc ? w[(size_t)c * kTaps + tap] : 0.f, 0.f, SplitScale<false>(field), h, l);
        uint8_t* to = out + ((size_t)column * blocks * kTaps + segment) * 2 * plane + (size_t)row * 128 +
                      (((k >> 3) ^ (row & 7)) << 4) + (k & 7) * 2;
        *reinterpret_cast<uint16_t*>(to) = (uint16_t)h;
        *reinterpret_cast<uint16_t*>(to + plane) = (uint16_t)l;
    }
}

template <int BN>
__global__ void __launch_bounds__(Cfg<BN>::kThreads, 1) conv_f32_patch_kernel(
        const __grid_constant__ PatchF32Params p) {
    using C = Cfg<BN>;
    constexpr int kBars = C::kBars, kGroup = C::kGroup, kGroups = kTaps / kGroup;
    constexpr int kEpilogueWarps = C::kEpilogueWarps;
    constexpr int kTmemColumns = kBars * kGroup * BN <= 256 ? 256 : 512;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* plane_full = (uint64_t*)smem;        // [2] converters -> MMA
    uint64_t* plane_empty = plane_full + 2;        // [2]
    // a group's MMAs may go: accumulators free (the epilogue), filter loaded (the
    // TMA); ... have retired (epilogue, producer)
    uint64_t* ready = plane_empty + 2;             // [kBars]
    uint64_t* done = ready + kBars;                // [kBars]
    uint64_t* drain_bar = done + kBars;
    uint64_t* exact_bars = drain_bar + 1;          // [2]
    uint32_t* tmem_slot = (uint32_t*)(exact_bars + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    ColumnStates* columns = (ColumnStates*)(tmem_slot + 2);
    LateTiles* late = reinterpret_cast<LateTiles*>(smem + C::kLateOff);
    const uint32_t late_a = smem_u32(late);
    float* factors = reinterpret_cast<float*>(smem + C::kFactorOff);  // [kFactorSets][kPixels]
    uint8_t* planes = smem + C::kFrontBytes;       // [2][hi, lo]
    uint8_t* ring_b = planes + C::kPlaneBytes;
    uint8_t* turned = ring_b + C::kBStages * C::kBBytes;  // [kEpilogueWarps][32 rows][kTurn columns]

    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    const int total_tiles = p.m_tiles * p.n_tiles;
    const int first_tile = (int)blockIdx.x, tile_step = (int)gridDim.x;

    if (threadIdx.x == 0) {
        for (int b = 0; b < 2; ++b) {
            mbar_init(&plane_full[b], kConverterWarps);
            mbar_init(&plane_empty[b], 1);
        }
        for (int t = 0; t < kBars; ++t) {
            mbar_init(&ready[t], kEpilogueWarps + 1);
            mbar_init(&done[t], 1);
        }
        mbar_init(drain_bar, 1);
        mbar_init(&exact_bars[0], 1);
        mbar_init(&exact_bars[1], 1);
        *abort_flag = 0;
        columns->reset();
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < sizeof(LateTiles) / 4)
        late->bits[threadIdx.x] = 0;
    if (warp == 1) {
        asm volatile(
                "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                        smem_u32(tmem_slot)),
                "r"(kTmemColumns)
                : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    const uint32_t ready_a = smem_u32(ready), done_a = smem_u32(done);

    auto give_up = [&](int code) {
        if (!*abort_flag) {
            *abort_flag = 1;
            atomicExch(p.status, code);
        }
    };

    if (warp == 0) {
        // ---------------- filter producer (a converged warp, one lane issues) ----------------
        const uint32_t leader = elect_one() ? 1u : 0u;
        const uint32_t ring_0 = smem_u32(ring_b);
        pdl_wait();  // from here on the kernel touches global memory
        pdl_release();
        uint32_t turn = 0;
        bool ok = true;
        const bool stays = p.n_tiles == 1 && p.blocks * kGroups <= C::kBStages;
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
            const uint8_t* from = p.filter + (size_t)(tile % p.n_tiles * p.blocks) * (kTaps * C::kTapBytes);
            for (int block = 0; block < p.blocks && ok; ++block) {
                for (int group = 0; group < kGroups; ++group, ++turn, from += C::kBBytes) {
                    // the stage's group before must have retired
                    const uint32_t before = turn - (uint32_t)C::kBStages;
                    if (turn >= (uint32_t)C::kBStages)
                        ok = mbar_wait_u32(done_a + 8 * (before % kBars), (before / kBars) & 1u, abort_flag);
                    if (!ok)
                        break;
                    const uint32_t bar = ready_a + 8 * (turn % kBars);
                    if (stays && turn >= (uint32_t)C::kBStages) {
                        if (leader)
                            mbar_arrive_u32(bar);
                        continue;
                    }
                    mbar_expect_tx_if(leader, bar, (uint32_t)C::kBBytes);
                    bulk_load_if(leader, ring_0 + (turn % C::kBStages) * C::kBBytes, from, C::kBBytes, bar);
                }
            }
        }
        if (!ok)
            give_up(ERR_PRODUCER_WAIT);
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer (the whole warp waits, one lane issues) ----------------
        // (Every wait's outcome is voted on, and the base of the tensor memory comes from one lane: the
        // control flow and the operands' descriptors are then the warp's and not its lanes', and an MMA is
        // issued sooner. 32 x 80 x 80 pixels, 64 -> 64: 65.9 -> 60.7 us.)
        const uint32_t leader = elect_one() ? 1u : 0u;
        constexpr uint32_t idesc = umma_idesc_f16(kBM, BN);
        // 128-byte swizzled K-major rows. B: 8-row groups 1024 bytes apart; A: patch rows, 10 pixels apart
        constexpr uint32_t kLow = 1u << 16;
        constexpr uint32_t kHigh = (1u << 14) | (2u << 29);
        constexpr uint32_t kBHigh = kHigh | (1024 / 16), kAHigh = kHigh | (kPW * 128 / 16);
        constexpr uint32_t kBPlane = C::kTapBytes / 2 / 16, kAPlane = kPlane / 16;
        const uint32_t plane_full_a = smem_u32(plane_full), plane_empty_a = smem_u32(plane_empty);
        const uint32_t a_first = ((smem_u32(planes) & 0x3FFFFu) >> 4) | kLow;
        const uint32_t b_first = ((smem_u32(ring_b) & 0x3FFFFu) >> 4) | kLow;
        uint32_t b_hi = b_first, phase = 0, plane_turn = 0;
        int slot = 0, t = 0;
        bool ok = true;
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
            for (int block = 0; block < p.blocks && ok; ++block, ++plane_turn) {
                const uint32_t buf = plane_turn & 1;
                ok = __all_sync(0xffffffffu,
                                mbar_wait_u32(plane_full_a + 8 * buf, (plane_turn >> 1) & 1u, abort_flag));
                if (!ok)
                    break;  // (the next wait may well succeed: filter and accumulators know nothing of the planes)
                const uint32_t a_block = a_first + buf * 2 * kAPlane;
                const int left = p.ic - block * kBlock;
                const int steps = left >= kBlock ? kBlock / 16 : (left + 15) / 16;
                for (int group = 0; group < kGroups; ++group) {
                    ok = __all_sync(0xffffffffu, mbar_wait_u32(ready_a + 8 * t, phase, abort_flag));
                    if (!ok)
                        break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    auto taps = [&](auto count) {
                        constexpr int kSteps = decltype(count)::value;
#pragma unroll
                        for (int i = 0; i < kGroup; ++i) {
                            const uint32_t d = tmem_base + (t * kGroup + i) * BN;
                            const int shift = kGroup == 3 ? group * kPW + i : group / 3 * kPW + group % 3;
                            const uint32_t a_hi = a_block + (uint32_t)(shift * (128 / 16));
                            const uint32_t a_lo = a_hi + kAPlane;
                            const uint32_t tap_hi = b_hi + i * (C::kTapBytes / 16), tap_lo = tap_hi + kBPlane;
                            // a K step of 16: 32 bytes inside the swizzled rows; the small products first
#pragma unroll
                            for (int k = 0; k < kSteps; ++k) {
                                umma_f16_ss(leader, d, a_lo + 2 * k, tap_hi + 2 * k, kAHigh, kBHigh, idesc, k != 0);
                                umma_f16_ss(leader, d, a_hi + 2 * k, tap_lo + 2 * k, kAHigh, kBHigh, idesc, 1);
                            }
                            umma_f16_ss<kLoShift>(leader, d, a_hi, tap_hi, kAHigh, kBHigh, idesc, 1);
#pragma unroll
                            for (int k = 1; k < kSteps; ++k)
                                umma_f16_ss(leader, d, a_hi + 2 * k, tap_hi + 2 * k, kAHigh, kBHigh, idesc, 1);
                        }
                    };
                    if (steps == 4)
                        taps(Number<4>());
                    else if (steps == 3)
                        taps(Number<3>());
                    else if (steps == 2)
                        taps(Number<2>());
                    else
                        taps(Number<1>());
                    umma_commit_if(leader, done_a + 8 * t);
                    b_hi += C::kBBytes / 16;
                    if (++slot == C::kBStages) {
                        slot = 0;
                        b_hi = b_first;
                    }
                    if (++t == kBars) {
                        t = 0;
                        phase ^= 1u;
                    }
                }
                if (ok)
                    umma_commit_if(leader, plane_empty_a + 8 * buf);
            }
        }
        if (!ok)
            give_up(ERR_MMA_WAIT);
        __syncwarp();
    } else if (warp >= 2 + kEpilogueWarps) {
        // ---------------- converters: fp32 patch -> hi and lo planes ----------------
        // Four lanes have a pixel; of every 16 channels each has four, so that a warp's loads are whole 64-byte
        // pieces. The next block's pixels are on their way while these are split. (Pixels in the order 0 2 4 6
        // 1 3 5 7: the 8-byte stores of half a warp then take all banks.)
        const int cw = warp - 2 - kEpilogueWarps;
        const int part = lane & 3, mine = (lane >> 2 & 3) * 2 + (lane >> 4) + cw * 8;
        constexpr int kTurns = (kPixels + 8 * kConverterWarps - 1) / (8 * kConverterWarps);
        const uint32_t plane_full_a = smem_u32(plane_full), plane_empty_a = smem_u32(plane_empty);
        uint32_t turn = 0, ordinal = 0;
        bool ok = true;
        pdl_wait();
        // this lane's channels of its pixel in turn i, zero beyond the image and the channels
        auto load = [&](const TilePos& at, int block, int i, float4 (&v)[4]) {
            const int px = mine + i * 8 * kConverterWarps;
            const int dy = px / kPW, dx = px - dy * kPW;
            const int y = at.y0 - 1 + dy, x = at.x0 - 1 + dx;
            const bool inside = px < kPixels && (unsigned)y < (unsigned)p.oh && (unsigned)x < (unsigned)p.ow;
            const int left = inside ? p.ic - block * kBlock - part * 4 : 0;
            const float* from =
                    p.src + (((size_t)at.img * p.oh + y) * p.ow + x) * p.src_pitch + block * kBlock + part * 4;
#pragma unroll
            for (int u = 0; u < 4; ++u)
                v[u] = 16 * u < left ? __ldcg(reinterpret_cast<const float4*>(from + 16 * u))
                                     : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        float4 v[kTurns][4];
        if (first_tile < total_tiles) {
            const TilePos at(first_tile, BN, p);
#pragma unroll
            for (int i = 0; i < kTurns; ++i)
                load(at, 0, i, v[i]);
        }
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step, ++ordinal) {
            // Operands that the planes do not hold put the tile off
            const bool strict = __any_sync(0xffffffffu, columns->is_strict(p.n_tiles == 1 ? 0 : tile % p.n_tiles));
            bool fits = true;
            LargestValues values;
            values.reset();
            for (int block = 0; block < p.blocks && ok; ++block, ++turn) {
                const uint32_t buf = turn & 1;
                const int left = p.ic - block * kBlock;
                const int steps = left >= kBlock ? kBlock / 16 : (left + 15) / 16;
                uint8_t* hi_plane = planes + buf * 2 * kPlane;
                float* factor = factors + (turn % C::kFactorSets) * kPixels;
                const bool same = block + 1 < p.blocks;  // the next block is of this tile
                const bool more = same || tile + tile_step < total_tiles;
                const TilePos then(same ? tile : tile + tile_step, BN, p);
                const int then_block = same ? block + 1 : 0;
                ok = mbar_wait_u32(plane_empty_a + 8 * buf, ((turn >> 1) & 1u) ^ 1u, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok)
                    break;
#pragma unroll
                for (int i = 0; i < kTurns; ++i) {
                    const int px = mine + i * 8 * kConverterWarps;
                    float most = 0.f;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        most = fmaxf(most, fmaxf(fmaxf(fabsf(v[i][u].x), fabsf(v[i][u].y)),
                                                 fmaxf(fabsf(v[i][u].z), fabsf(v[i][u].w))));
                    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 1));
                    most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 2));
                    const uint32_t field = scale_field(most);
                    const SplitScale<false> scale(field);
                    values.take(most);
                    if (strict) {
                        uint32_t least = 0xffffffffu;
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            least = min(min(least, min(magnitude_0_last(v[i][u].x), magnitude_0_last(v[i][u].y))),
                                        min(magnitude_0_last(v[i][u].z), magnitude_0_last(v[i][u].w)));
                        fits = fits && least >= least_magnitude(field);
                    }
                    if (px < kPixels) {
                        if (part == 0)
                            factor[px] = field_to_float(pixel_factor_field(field));
                        // 16-byte unit u of pixel p sits at unit u ^ (p & 7) of its row
                        uint8_t* row = hi_plane + px * 128 + (part & 1) * 8;
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (u >= steps)
                                break;
                            uint2 hi, lo;
                            split_f16(v[i][u].x, v[i][u].y, scale, hi.x, lo.x);
                            split_f16(v[i][u].z, v[i][u].w, scale, hi.y, lo.y);
                            uint8_t* to = row + (((u * 2 + (part >> 1)) ^ (px & 7)) << 4);
                            *reinterpret_cast<uint2*>(to) = hi;
                            *reinterpret_cast<uint2*>(to + kPlane) = lo;
                        }
                    }
                    if (more)
                        load(then, then_block, i, v[i]);
                }
                if (block + 1 == p.blocks)
                    put_tile_off_if(!(fits && values.fit()), late_a, ordinal);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0)
                    mbar_arrive_u32(plane_full_a + 8 * buf);
            }
        }
        if (!ok)
            give_up(ERR_PRODUCER_WAIT);
        __syncwarp();
    } else {
        // ---------------- epilogue: warps from 2 on, TMEM lanes 32 * (warp % 4) .. ----------------
        const int q = warp & 3;
        const int row = q * 32 + lane;
        const int py = row >> 3, px = row & 7;
        constexpr int kCols = C::kCols;
        const int col0 = (warp - 2) / 4 * kCols;  // this warp's columns
        const uint32_t turned_w = smem_u32(turned) + (warp - 2) * C::kTurnBytes;
        float* channels = reinterpret_cast<float*>(smem + C::kChannelOff) + col0;  // [2][factor, bias][BN]
        uint32_t turn = 0, plane_turn = 0;
        int set = 1;
        bool ok = true;
        if (lane == 0) {  // all accumulators are free
            for (int t = 0; t < kBars; ++t)
                mbar_arrive(&ready[t]);
        }
        pdl_wait();  // before the first read of z and the first store
        find_column_states<32 * kEpilogueWarps, 1>(p.factor, p.oc, BN, (int)threadIdx.x - 64, columns, &late->any);
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
            const TilePos at(tile, BN, p);
            const int oy = at.y0 + py, ox = at.x0 + px;
            const bool valid = oy < p.oh && ox < p.ow;
            const size_t m = ((size_t)at.img * p.oh + oy) * p.ow + ox;
            if (p.n_tiles > 1 || tile == first_tile) {
                // (the warps of the same columns write the same numbers to the same place)
                set ^= 1;
#pragma unroll
                for (int j = lane; j < kCols; j += 32) {
                    const int ch = at.n0 + col0 + j;
                    channels[set * 2 * BN + j] =
                            ch < p.oc ? channel_factor(__float_as_uint(__ldg(p.factor + ch))) : 0.f;
                    channels[set * 2 * BN + BN + j] = p.ep.bias && ch < p.oc ? __ldg(p.ep.bias + ch) : 0.f;
                }
            }
            if (p.ep.z && valid) {
                const float* zin = p.ep.z + m * p.ep.z_pitch + at.n0 + col0;
#pragma unroll
                for (int j = 0; j < kCols; j += 32)
                    if (at.n0 + col0 + j < p.oc)
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(zin + j));
            }
            // running fp32 sums of this thread's accumulators over the tile's segments
            float sum[kCols];
#pragma unroll
            for (int j = 0; j < kCols; ++j)
                sum[j] = 0.f;
            const uint32_t lane_base =
                    tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)col0;
            for (int block = 0; block < p.blocks && ok; ++block, ++plane_turn) {
                const float* factor = factors + (plane_turn % C::kFactorSets) * kPixels + py * kPW + px;
                for (int group = 0; group < kGroups; ++group, ++turn) {
                    ok = mbar_wait_u32(done_a + 8 * (turn % kBars), (turn / kBars) & 1u, abort_flag);
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) {
                        give_up(ERR_EPILOGUE_WAIT);
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    // (Each load is waited for in the statement that issues it: with a load in flight
                    // across other code, a register that it has yet to write must never be spilled, and
                    // with this many sums nothing guarantees that.)
                    const uint32_t d = lane_base + (turn % kBars) * (kGroup * BN);
                    if constexpr (BN == 32) {
                        uint32_t v[48];
                        tmem_ld16x3(d, d + BN, d + 2 * BN, v);
#pragma unroll
                        for (int i = 0; i < 3; ++i) {
                            const float f = factor[group * kPW + i];
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                sum[j] = __fmaf_rn(__uint_as_float(v[16 * i + j]), f, sum[j]);
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < kGroup; ++i) {
                            const float f = factor[kGroup == 3 ? group * kPW + i : group / 3 * kPW + group % 3];
#pragma unroll
                            for (int c = 0; c < kCols / 16; ++c) {
                                uint32_t v[16];
                                tmem_ld16(d + (uint32_t)(i * BN + 16 * c), v);
#pragma unroll
                                for (int j = 0; j < 16; ++j)
                                    sum[16 * c + j] = __fmaf_rn(__uint_as_float(v[j]), f, sum[16 * c + j]);
                            }
                        }
                    }
                    // the warp's accumulators are in registers: hand the set back
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(&ready[turn % kBars]);
                }
            }
            if (!ok)
                break;
            if (at.n0 + col0 < p.oc) {
                const float* channel = channels + set * 2 * BN;
                const int y0 = at.y0 + q * 4;
                const PatchRows rows{p, ((size_t)at.img * p.oh + y0) * p.ow + at.x0, y0, at.x0};
                store_f32_rows<kCols, C::kTurn, true>(sum, p.ep, turned_w, channel, channel + BN, rows,
                                                      at.n0 + col0);
            }
        }
    }

    // ---------------- the tiles put off, teardown ----------------
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*(volatile uint32_t*)&late->any != 0 && !*abort_flag) {
        exact_tiles<BN>(p, late, columns, planes, tmem_base, exact_bars, abort_flag);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
    }
    if (*abort_flag) {
        if (warp == 1 && lane == 0) {
            umma_commit(drain_bar);
            const long long t0 = clock64();
            while (!mbar_try_wait(drain_bar, 0)) {
                if (clock64() - t0 > kWaitCycles) {
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
                     "r"(kTmemColumns)
                     : "memory");
    }
}

template <int BN>
int launch_bn(PatchF32Params& p, size_t out_bytes, cudaStream_t st) {
    static KernelReady ready;
    if (!ready.smem(conv_f32_patch_kernel<BN>, Cfg<BN>::kDynamic))
        return check_launch("conv_f32_patch smem attribute");
    const int total = p.m_tiles * p.n_tiles;
    const int grid = total < sm_count() ? total : sm_count();
    if (tuning().debug)
        fprintf(stderr, "conv_f32_patch<%d>: grid %d tiles %d x %d blocks %d smem %d\n", BN, grid, p.m_tiles,
                p.n_tiles, p.blocks, Cfg<BN>::kDynamic);
    launch_pdl(Writes{p.ep.dst, out_bytes}, conv_f32_patch_kernel<BN>, dim3(grid),
               dim3(Cfg<BN>::kThreads), (size_t)Cfg<BN>::kDynamic, st, p);
    return check_launch("conv_f32_patch");
}

int tile_columns(int oc) {
    return oc <= 32 ? 32 : oc <= 64 ? 64 : 128;
}

}  // namespace

// floats of the planes of such a filter, behind which its channel words lie, and of both
size_t conv_f32_patch_words_at(const ConvF32Args& a) {
    const int bn = tile_columns(a.oc);
    const size_t channels = (size_t)(a.oc + bn - 1) / bn * bn, blocks = (a.ic + kBlock - 1) / kBlock;
    return channels * blocks * kBlock * kTaps;
}
size_t conv_f32_patch_filter_floats(const ConvF32Args& a) {
    const int bn = tile_columns(a.oc);
    return conv_f32_patch_words_at(a) + (size_t)(a.oc + bn - 1) / bn * bn;
}

int launch_conv_f32_pack_filter_patch(
        const ConvF32Args& a, const float* flt_oihw, float* out, cudaStream_t st) {
    const int bn = tile_columns(a.oc), blocks = (a.ic + kBlock - 1) / kBlock;
    const int channels = (a.oc + bn - 1) / bn * bn;
    pack_filter_patch_kernel<<<channels, 256, 0, st>>>(flt_oihw, (uint8_t*)out,
                                                       (uint32_t*)out + conv_f32_patch_words_at(a), a.oc, a.ic, blocks, bn);
    return check_launch("pack_filter_f32_patch");
}

// Does a packed filter hold the planes of this kernel? (By the filter alone, see conv_f32_split_planes, and
// what it was packed for.)
bool conv_f32_patch_planes(const ConvF32Args& a) {
    return (a.forms & F32_PATCH_PLANES) && conv_f32_split_planes(a) && a.kh == 3 && a.kw == 3;
}
// ... and may the ConvBias take it?
bool conv_f32_patch_shape(const ConvF32Args& a) {
    return conv_f32_patch_planes(a) && a.sh == 1 && a.sw == 1 && a.ph == 1 && a.pw == 1;
}

// ... and is it the faster one then? Both kernels' time goes with the tiles of the busiest SM; a patch that is not
// full is paid for in full. What a patch takes beside an im2col tile of the same columns and channels, in
// percent, was measured as what one more on every SM costs, full patches, 200 to 1600 of them (us, im2col -> patches at
// 400 and 1600; SILU or no activation alike):
//   128 columns: 128 channels 54.0 -> 43.5, 202 -> 166; 64 channels 31.6 -> 26.3, 110 -> 99; 32 and 16: none better
//    64 columns:  64 channels 25.9 -> 17.9, 87 -> 63; 32 channels 16.8 -> 14.1, 51.6 -> 41.9; 16: none better
//    32 columns:  64 channels 21.9 -> 15.5, 71 -> 45; 32 channels 13.1 -> 11.9, 37.6 -> 31.9; 16: 10.3 -> 9.7, 28.9 -> 25.3
// That is one layer over and over. In a network a patch kernel takes some 3 us more, which im2col kernels, of
// which the layers around are, do not (kStart, in the clocks of conv_f32_tile_clocks). The detector with every
// layer that is the faster one by itself, us beside none of them: one image of 256 x 256 +4.0, 416 x 416 +2.8,
// 480 x 480 +4.1, two of 320 x 320 +5.1, four of 416 x 416 +4.7, of 640 x 640 -40; by this rule +0.3, -0.2, -0.2,
// -0.2, -5.8 and -39.
// im2col tiles of at most half the SMs are split over clusters and stay (1 x 80 x 80, 50 of each: 64 -> 64 9.2 and
// 9.2, 16 -> 32 5.2 and 5.6).
bool conv_f32_patch_pays(const ConvF32Args& a) {
    const int bn = tile_columns(a.oc);
    const long long sms = sm_count(), columns = (a.oc + bn - 1) / bn;
    const long long patches = (long long)a.n * ((a.oh + kTH - 1) / kTH) * ((a.ow + kTW - 1) / kTW) * columns;
    if (patches > sms * kExactTiles)
        return false;
    if (tuning().f32_patch != 1)
        return tuning().f32_patch == 2;
    const long long tiles = ((long long)a.m + kBM - 1) / kBM * columns;
    const int percent = a.ic > 32 ? (bn == 128 ? 84 : bn == 64 ? 66 : 60)
                        : a.ic > 16 ? (bn == 128 ? 100 : bn == 64 ? 80 : 80)
                                    : (bn == 32 ? 83 : 100);
    if (percent == 100 || 2 * tiles <= sms)
        return false;
    constexpr long long kStart = 4000;
    const long long tile = conv_f32_tile_clocks(a, bn);
    return (patches + sms - 1) / sms * percent * tile + 100 * kStart < (tiles + sms - 1) / sms * 100 * tile;
}

int launch_conv_f32_patch(
        const ConvF32Args& a, const float* src, const float* planes, const float* weights, const float* bias,
        const float* z, float* dst, cudaStream_t st) {
    const int bn = tile_columns(a.oc);
    PatchF32Params p;
    p.n = a.n;
    p.oh = a.oh;
    p.ow = a.ow;
    p.oc = a.oc;
    p.ic = a.ic;
    p.src = src;
    p.src_pitch = a.src_pitch;
    p.blocks = (a.ic + kBlock - 1) / kBlock;
    p.tiles_y = (a.oh + kTH - 1) / kTH;
    p.tiles_x = (a.ow + kTW - 1) / kTW;
    p.m_tiles = a.n * p.tiles_y * p.tiles_x;
    p.n_tiles = (a.oc + bn - 1) / bn;
    p.ep.oc = a.oc;
    p.ep.act = a.act;
    p.ep.bias = bias;
    p.ep.z = z;
    p.ep.z_pitch = a.z_pitch;
    p.ep.dst = dst;
    p.ep.dst_pitch = a.dst_pitch;
    p.filter = reinterpret_cast<const uint8_t*>(planes);
    p.factor = planes + conv_f32_patch_words_at(a);
    p.exact = conv_f32_exact_operands(a, src, weights, false);
    p.status = device_status_word(st);
    if (!p.status)
        return ST_MALLOC;
    const size_t out_bytes = (size_t)a.m * a.dst_pitch * 4;
    return bn == 32   ? launch_bn<32>(p, out_bytes, st)
           : bn == 64 ? launch_bn<64>(p, out_bytes, st)
                      : launch_bn<128>(p, out_bytes, st);
}

}  // namespace mb200
