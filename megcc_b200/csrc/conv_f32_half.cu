// fp32 ConvBias / MatrixMul on the sm_100a tensor cores with fp32-level accuracy, wide layers: tiles of
// 128 pixels x 128 channels, operands split into two fp16 values. (conv_f32.cu splits into two tf32 values
// and has everything else: narrow tiles, tiles split over a cluster, rows of 64 bytes.)
//
// Every operand is scaled by a power of two and split, v s = hi + 2^-12 lo (conv_f32_split.cuh), and a product
// is three passes of tcgen05.mma kind::f16,
//     2^-12 (lo*hi + hi*lo) + hi*hi                                    (lo*lo is < 2^-22)
// which leaves a relative error of a few 2^-23 per product, the order of fp32 itself: the same 11 + 11
// bits as with tf32 at half the tensor time and half the filter's bytes. fp16 has few exponents, so the
// scale follows the data: one per pixel and 64 elements of K for the activation, from the largest of them,
// one per output channel for the filter. Elements down to 2^-30 of the largest keep their bits; tiles whose
// operands lie further apart are put off and taken from tf32 planes at the kernel's end
// (conv_f32_exact.cuh). A K segment of 64 elements has accumulators of its own, whose sum is multiplied by the
// pixel's factor when it is added up.
//
// The tensor core adds into its accumulator with truncation (see conv_f32.cu), so chains are kept short
// here too: a segment's eight small products come first (their sum goes into the main one 2^-12 times, so its
// truncation does not matter), then four K = 16 steps of hi*hi; the epilogue warps add finished segments
// into fp32 registers with round-to-nearest.
//
// What bounds a tile is the SM's shared-memory port: a segment moves 144 KB through it (TMA writes 64, the
// converters' reads 32, B reads of twelve MMAs 48), 1152 clocks at 128 bytes a clock against 768 of tensor
// time; with tf32 it is 224 KB and 1792 against 1536. Measured 1750 to 1950 clocks a segment (tf32:
// 2300): the converters' chain of a segment (wait, read, largest value, split, write) is 1370, and with
// the rings three segments deep it and the TMA's round trip overlap only in part. Per call, tf32 and here: 32 x 80 x 80 pixels, 128 -> 128
// 3x3 282 and 224 us, 1x1 59.7 and 47.0, 128 -> 256 3x3/2 137 and 109, a 2048^3 product with its preparation 93 and 80.
// Against 64 bits the results are no further off (2-norm, N(0,1) operands: K = 1152 2.1e-7 and 1.6e-7,
// K = 4096 2.3e-7 and 2.0e-7; K = 1152 with one channel 2^16 to 2^40 up under weights as far down 2.1e-7 and 1.7e-7).
// Narrower tiles do not gain: their TMA rows (4 clocks each) are the same with either split.
//
// Structure: persistent CTAs, warp 0 TMA producer (im2col or plain matrix rows), warp 1 MMA issuer and
// TMEM owner, warps 2..9 epilogue, warps 10..17 converters (fp32 tile -> planes in tensor memory, half a
// segment of one pixel per thread), bounded waits.
//
// Replaces, for the fp32 configurations, the reference's im2col + 4x12 SIMD GEMM
// (compiler/lib/KernelGen/GeneralIntrinsic/ConvKernel/Fp32Im2col.cpp:122-217,
// GeneralIntrinsic/MatMulKernel/Fp32MatMulM4N12.cpp:8-160).
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
constexpr int kSegK = 64;     // K elements that share an accumulator and a pixel's scale
constexpr int kBN = 128;
constexpr int kChans = 32;    // floats per row of A (128 bytes); two rows make a segment
constexpr int kMaxAStages = 8;
constexpr int kTStages = 4;   // segments of A planes in tensor memory
constexpr int kTCols = kSegK; // columns of one: two planes, two fp16 per column
constexpr int kAccCols = 2 * kBN;
static_assert(kAccCols + kTStages * kTCols <= 512, "tensor memory");
constexpr int kABytes = kBM * kChans * 4;
constexpr int kBBytes = 2 * kBN * kSegK * 2;  // both planes of a filter segment
constexpr int kEpilogueWarps = 8, kConverterWarps = 8;
constexpr int kThreads = 64 + 32 * (kEpilogueWarps + kConverterWarps);
// shared memory in front of the tiles: barriers and which tile columns are wide or loose; a bit for each tile that
// is put off; the pixels' factors of the last eight segments; the
// converters' largest values (two segments, two halves); each epilogue warp's bias and channel factors
constexpr int kLateOff = 448, kFactorOff = 1024, kMostOff = kFactorOff + 8 * kBM * 4;
static_assert(kLateOff + sizeof(LateTiles) <= kFactorOff, "the list of tiles");
constexpr int kBiasOff = kMostOff + 4 * kBM * 4;
constexpr int kTurn = 16;     // columns of a result turned round at a time
constexpr int kTurnOff = kBiasOff + kEpilogueWarps * kBN / 2 * 8;
constexpr int kFrontBytes = (kTurnOff + kEpilogueWarps * 32 * kTurn * 4 + 1023) / 1024 * 1024;
constexpr int kTileBudget = 227 * 1024 - 1024 - kFrontBytes;  // (1024: alignment)
constexpr int kDynamic = 227 * 1024;

// A operand (two fp16 per column) in tensor memory, B in shared memory (descriptor as its two words);
// issued by the lane whose `leader` is non-zero. SHIFT: what is in the accumulator counts 2^-SHIFT times
template <int SHIFT = 0>
__device__ __forceinline__ void umma_f16_ta(
        uint32_t leader, uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi,
        uint32_t idesc, uint32_t accumulate) {
    asm volatile(
            "{\n\t.reg .pred p, q;\n\t.reg .b64 d;\n\t"
            "mov.b64 d, {%2, %3};\n\t"
            "setp.ne.b32 p, %5, 0;\n\tsetp.ne.b32 q, %6, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d, %4, p, %7;\n\t}" ::"r"(tmem_d),
            "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(leader), "n"(SHIFT)
            : "memory");
}

// 8 columns of this warp's 32 TMEM lanes <- registers (complete after tcgen05.wait::st)
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
            "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
            : "memory");
}

// ------------------------------------------------------------------------------------------
// filter packing (load time)
// ------------------------------------------------------------------------------------------
// fp16 planes [2][OC][KH][KW][ICp] (hi, lo), zero-filled beyond IC, then a word per OC (channel_word)
struct Planes {
    uint16_t *hi, *lo;
    uint32_t* word;
};
__device__ __forceinline__ Planes planes_at(float* out, size_t plane) {
    uint16_t* hi = reinterpret_cast<uint16_t*>(out);
    return Planes{hi, hi + plane, reinterpret_cast<uint32_t*>(out + plane)};
}

// OIHW fp32 -> the planes, a block per output channel
__global__ void __launch_bounds__(256) pack_filter_half_kernel(
        const float* __restrict__ src, float* __restrict__ out, int oc, int ic, int icp, int kh,
        int kw) {
    __shared__ Magnitudes shared[8];
    const int taps = kh * kw, o = blockIdx.x;
    const float* w = src + (size_t)o * ic * taps;
    Magnitudes of = Magnitudes::none();
    for (int i = threadIdx.x; i < ic * taps; i += 256)
        of.take(w[i]);
    of = block_magnitudes(of, shared);
    const uint32_t field = scale_field(of.largest);
    const Planes d = planes_at(out, (size_t)oc * taps * icp);
    if (threadIdx.x == 0)
        d.word[o] = of.word();
    for (int i = threadIdx.x; i < taps * icp; i += 256) {
        const int tap = i / icp, c = i - tap * icp;
        uint32_t h, l;
        split_f16(c < ic ? w[(size_t)c * taps + tap] : 0.f, 0.f, SplitScale<false>(field), h, l);
        d.hi[(size_t)o * taps * icp + i] = (uint16_t)h;
        d.lo[(size_t)o * taps * icp + i] = (uint16_t)l;
    }
}

// [K][N] fp32 (the second operand of a matrix product) -> the same [N][Kp], 32 columns per cluster of
// kPackParts blocks, which share the rows: the columns' largest values, exchanged over the cluster, then
// the planes, a 32 x 64 tile at a time through shared memory. The second read comes from the L2, so
// HBM moves 8 bytes per element.
constexpr int kPackParts = 8;
__global__ void __launch_bounds__(256) pack_matrix_half_kernel(
        const float* __restrict__ src, float* __restrict__ out, int k, int n, int kp) {
    // (a column's magnitudes, 16 bytes each: other blocks of the cluster read them)
    __shared__ __align__(16) float found[32][4];
    __shared__ Magnitudes part[8][33];
    __shared__ float tile[64][33];
    const int lane = threadIdx.x & 31, row = threadIdx.x >> 5;
    const int n0 = (int)(blockIdx.x / kPackParts) * 32;
    const int rank = (int)cluster_rank();
    const int blocks = (kp + 63) / 64;
    const int c = n0 + lane;
    // rows of this block: every kPackParts-th 64
    Magnitudes v = Magnitudes::none();
    if (c < n) {
        for (int b = rank; b < blocks; b += kPackParts) {
            float x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int r = b * 64 + row + 8 * j;
                x[j] = __ldg(src + (size_t)(r < k ? r : 0) * n + c);  // (a value twice does not matter)
            }
#pragma unroll
            for (int j = 0; j < 8; ++j)
                v.take(x[j]);
        }
    }
    part[row][lane] = v;
    __syncthreads();
    if (row == 0) {
#pragma unroll
        for (int j = 1; j < 8; ++j)
            v.take(part[j][lane]);
        found[lane][0] = v.largest;
        found[lane][1] = v.least;
        found[lane][2] = v.least_nonzero;
    }
    __syncthreads();
    cluster_arrive();
    cluster_wait();
    // (a thread's column for the writes: four threads of a column's row)
    const int col = threadIdx.x >> 3, kq = (threadIdx.x & 7) * 8;
    v = Magnitudes::none();
    for (int i = 0; i < kPackParts; ++i) {
        const uint4 w = ld_cluster_v4(smem_u32(found[col]), i);
        v.take(Magnitudes{__uint_as_float(w.x), __uint_as_float(w.y), __uint_as_float(w.z)});
    }
    cluster_arrive();
    const uint32_t field = scale_field(v.largest);
    const SplitScale<true> scale(field);
    const Planes d = planes_at(out, (size_t)n * kp);
    const int cw = n0 + col;
    if (rank == 0 && cw < n && kq == 0)
        d.word[cw] = v.word();
    for (int b = rank; b < blocks; b += kPackParts) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int r = b * 64 + row + 8 * j;
            tile[row + 8 * j][lane] = r < k && c < n ? __ldg(src + (size_t)r * n + c) : 0.f;
        }
        __syncthreads();
        const int k0 = b * 64 + kq;
        if (cw < n && k0 < kp) {  // (kp is a multiple of 16)
            float x[8];
            uint32_t h[4], l[4];
#pragma unroll
            for (int j = 0; j < 8; ++j)
                x[j] = tile[kq + j][col];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                split_f16(x[2 * j], x[2 * j + 1], scale, h[j], l[j]);
            const size_t at = (size_t)cw * kp + k0;
            *reinterpret_cast<uint4*>(d.hi + at) = make_uint4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<uint4*>(d.lo + at) = make_uint4(l[0], l[1], l[2], l[3]);
        }
        __syncthreads();
    }
    cluster_wait();  // nobody leaves while its values may still be read
}

// ------------------------------------------------------------------------------------------
// the kernel
// ------------------------------------------------------------------------------------------
// rows that follow one another
struct RowPixel {
    int m0, m_total, oh, ow;
    __device__ __forceinline__ ExactPixel operator()(int row) const {
        const int m = m0 + row, img = m / (oh * ow), rem = m - img * (oh * ow), y = rem / ow;
        return ExactPixel{img, y, rem - y * ow, m < m_total};
    }
};

struct HalfConvParams {
    int m_total, oc, oh, ow;
    int cblocks;      // 32-channel rows per tap
    int taps_w;
    int k_iters;      // rows of the K loop
    int segs;         // segments: two rows each, the last may be one
    int sh, sw, base_h, base_w;
    int m_tiles, n_tiles;
    int a_tiled;      // 1x1, stride 1, no padding: A is the plain matrix [pixels][channels]
    int a_stages, b_stages;  // depth of the rings: rows of A (even), segments of B (at most kTStages)
    int b_resident;   // 1: the whole filter sits in shared memory
    F32Epilogue ep;
    const float* factor;  // per output channel: what a unit of the accumulated sums stands for (channel_word)
    ExactOperands exact;
    int* status;
    __device__ __forceinline__ RowPixel pixel(int tile) const {
        return RowPixel{tile / n_tiles * kBM, m_total, oh, ow};
    }
};

__global__ void __launch_bounds__(kThreads, 1) conv_f32_half_kernel(
        const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
        const __grid_constant__ HalfConvParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* a_full = (uint64_t*)smem;            // [kMaxAStages] TMA -> converters
    uint64_t* a_empty = a_full + kMaxAStages;      // [kMaxAStages] converters -> TMA
    // One barrier per segment says that its MMAs may go: planes written (the converters), accumulators free
    // (the epilogue, for the segment two on), filter loaded (the TMA); one that they have retired: for the
    // epilogue, for the converters (planes of the segment four on), for the producer (filter ring).
    // Each wait and each commit of the issuing warp shows as idle tensor time, 60 to 100 clocks.
    uint64_t* ready = a_empty + kMaxAStages;       // [kTStages]
    uint64_t* done = ready + kTStages;             // [kTStages]
    uint64_t* b_full = done + kTStages;            // a resident filter
    uint64_t* drain_bar = b_full + 1;
    uint64_t* exact_bars = drain_bar + 1;          // [2]
    uint32_t* tmem_slot = (uint32_t*)(exact_bars + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    ColumnStates* columns = (ColumnStates*)(tmem_slot + 2);
    LateTiles* late = reinterpret_cast<LateTiles*>(smem + kLateOff);
    const uint32_t late_a = smem_u32(late);
    float* pixel_factor = reinterpret_cast<float*>(smem + kFactorOff);  // [8][kBM]
    float* half_most = reinterpret_cast<float*>(smem + kMostOff);       // [2][2][kBM]
    uint8_t* tiles_b = smem + kFrontBytes;  // resident filter or ring of segments
    uint8_t* ring_a = tiles_b + (p.b_resident ? p.segs : p.b_stages) * kBBytes;

    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    const int total_tiles = p.m_tiles * p.n_tiles;
    const int first_tile = (int)blockIdx.x, tile_step = (int)gridDim.x;
    const int my_tiles =
            first_tile < total_tiles ? (total_tiles - 1 - first_tile) / tile_step + 1 : 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kMaxAStages; ++s) {
            mbar_init(&a_full[s], 1);
            mbar_init(&a_empty[s], kConverterWarps / 2);  // the half that reads the row
        }
        for (int t = 0; t < kTStages; ++t) {
            mbar_init(&ready[t], kConverterWarps + kEpilogueWarps + (p.b_resident ? 0 : 1));
            mbar_init(&done[t], 1);
        }
        mbar_init(b_full, 1);
        mbar_init(drain_bar, 1);
        mbar_init(&exact_bars[0], 1);
        mbar_init(&exact_bars[1], 1);
        *abort_flag = 0;
        columns->reset();
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    } else if (threadIdx.x == 32 * 2) {
        tma_prefetch_map(&map_a);
        tma_prefetch_map(&map_b);
    }
    if (threadIdx.x < sizeof(LateTiles) / 4)
        late->bits[threadIdx.x] = 0;
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
    const uint32_t ready_a = smem_u32(ready), done_a = smem_u32(done);

    auto give_up = [&](int code) {
        if (!*abort_flag) {
            *abort_flag = 1;
            atomicExch(p.status, code);
        }
    };

    if (warp == 0) {
        // ---------------- TMA producer (a converged warp, one lane issues) ----------------
        const uint32_t leader = elect_one() ? 1u : 0u;
        const uint32_t a_full_a = smem_u32(a_full), a_empty_a = smem_u32(a_empty);
        const uint32_t ring_a0 = smem_u32(ring_a), ring_b0 = smem_u32(tiles_b);
        const int pixels = p.oh * p.ow;
        pdl_wait();  // from here on the kernel touches global memory
        pdl_release();
        if (p.b_resident) {
            const uint32_t bar = smem_u32(b_full);
            mbar_expect_tx_if(leader, bar, (uint32_t)(p.segs * kBBytes));
            for (int g = 0; g < p.segs; ++g) {
                const uint32_t b = ring_b0 + g * kBBytes;
                tma_load_2d_if(leader, b, &map_b, bar, g * kSegK, 0);
                tma_load_2d_if(leader, b + kBBytes / 2, &map_b, bar, g * kSegK, p.oc);
            }
        }
        int sa = 0, sb = 0;
        uint32_t a_parity = 1, turn = 0;
        bool ok = true;
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
            const int tile_n = tile % p.n_tiles, tile_m = tile / p.n_tiles;
            const int m0 = tile_m * kBM, n0 = tile_n * kBN;
            const int img = m0 / pixels, rem = m0 - img * pixels;
            const int oy = rem / p.ow, ox = rem - oy * p.ow;
            const int base_w = ox * p.sw + p.base_w, base_h = oy * p.sh + p.base_h;
            int cb = 0, fx = 0, fy = 0;
            for (int g = 0; g < p.segs && ok; ++g) {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    ok = mbar_wait_u32(a_empty_a + 8 * sa, a_parity, abort_flag);
                    if (!ok)
                        break;
                    const uint32_t bar = a_full_a + 8 * sa, slot = ring_a0 + sa * kABytes;
                    // (a row that the last segment does not have keeps its turn of the ring: a slot
                    // always belongs to the same half of the converters)
                    const bool row = g * 2 + j < p.k_iters;
                    mbar_expect_tx_if(leader, bar, row ? (uint32_t)kABytes : 0u);
                    if (row) {
                        if (p.a_tiled)
                            tma_load_2d_if(leader, slot, &map_a, bar, cb * kChans, m0);
                        else
                            tma_load_im2col_4d_if(leader, slot, &map_a, bar, cb * kChans, base_w,
                                                  base_h, img, (uint16_t)fx, (uint16_t)fy);
                        if (++cb == p.cblocks) {
                            cb = 0;
                            if (++fx == p.taps_w) {
                                fx = 0;
                                ++fy;
                            }
                        }
                    }
                    if (++sa == p.a_stages) {
                        sa = 0;
                        a_parity ^= 1u;
                    }
                }
                if (ok && !p.b_resident) {
                    // the slot's segment before must have retired (the ring has no more slots than there
                    // are barriers)
                    const uint32_t before = turn - (uint32_t)p.b_stages;
                    if (turn >= (uint32_t)p.b_stages)
                        ok = mbar_wait_u32(done_a + 8 * (before % kTStages), (before / kTStages) & 1u,
                                           abort_flag);
                    if (!ok)
                        break;
                    const uint32_t bar = ready_a + 8 * (turn % kTStages), b = ring_b0 + sb * kBBytes;
                    ++turn;
                    mbar_expect_tx_if(leader, bar, (uint32_t)kBBytes);
                    tma_load_2d_if(leader, b, &map_b, bar, g * kSegK, n0);
                    tma_load_2d_if(leader, b + kBBytes / 2, &map_b, bar, g * kSegK, n0 + p.oc);
                    if (++sb == p.b_stages)
                        sb = 0;
                }
            }
        }
        if (!ok)
            give_up(ERR_PRODUCER_WAIT);
        __syncwarp();
    } else if (warp == 1) {
        // ---------------- MMA issuer (the whole warp waits, one lane issues) ----------------
        const uint32_t leader = elect_one() ? 1u : 0u;
        constexpr uint32_t idesc = umma_idesc_f16(kBM, kBN);
        // 128-byte swizzled K-major rows: 8-row groups 1024 bytes apart
        constexpr uint64_t kDesc = ((uint64_t)1 << 16) | ((uint64_t)(1024 / 16) << 32) |
                                   ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
        constexpr uint32_t kDescHi = (uint32_t)(kDesc >> 32);
        constexpr uint32_t kPlane = kBBytes / 2 / 16;
        const int slots = p.b_resident ? p.segs : p.b_stages;
        const uint32_t b_first = ((smem_u32(tiles_b) & 0x3FFFFu) >> 4) | (uint32_t)kDesc;
        const int last_steps = (p.k_iters * kChans - (p.segs - 1) * kSegK) / 16;
        uint32_t b_hi = b_first, phase = 0, buf = 0;
        int slot = 0, t = 0;
        bool ok = !p.b_resident || mbar_wait(b_full, 0, abort_flag);
        for (int tile = 0; tile < my_tiles && ok; ++tile) {
            for (int g = 0; g < p.segs; ++g) {
                ok = mbar_wait_u32(ready_a + 8 * t, phase, abort_flag);
                if (!ok)
                    break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem_base + buf * kBN;
                const uint32_t a_hi = tmem_base + kAccCols + (uint32_t)(t * kTCols);
                const uint32_t a_lo = a_hi + kTCols / 2, b_lo = b_hi + kPlane;
                const int steps = g + 1 == p.segs ? last_steps : kSegK / 16;
                // a K step of 16: 8 columns of A, 32 bytes inside B's swizzled row (+2 in the
                // descriptor's 16-byte address units)
                if (steps == kSegK / 16) {
#pragma unroll
                    for (int k = 0; k < kSegK / 16; ++k) {
                        umma_f16_ta(leader, d, a_lo + 8 * k, b_hi + 2 * k, kDescHi, idesc, k != 0);
                        umma_f16_ta(leader, d, a_hi + 8 * k, b_lo + 2 * k, kDescHi, idesc, 1);
                    }
                    umma_f16_ta<kLoShift>(leader, d, a_hi, b_hi, kDescHi, idesc, 1);
#pragma unroll
                    for (int k = 1; k < kSegK / 16; ++k)
                        umma_f16_ta(leader, d, a_hi + 8 * k, b_hi + 2 * k, kDescHi, idesc, 1);
                } else {
                    for (int k = 0; k < steps; ++k) {
                        umma_f16_ta(leader, d, a_lo + 8 * k, b_hi + 2 * k, kDescHi, idesc, k != 0);
                        umma_f16_ta(leader, d, a_hi + 8 * k, b_lo + 2 * k, kDescHi, idesc, 1);
                    }
                    umma_f16_ta<kLoShift>(leader, d, a_hi, b_hi, kDescHi, idesc, 1);
                    for (int k = 1; k < steps; ++k)
                        umma_f16_ta(leader, d, a_hi + 8 * k, b_hi + 2 * k, kDescHi, idesc, 1);
                }
                umma_commit_if(leader, done_a + 8 * t);
                b_hi += kBBytes / 16;
                if (++slot == slots) {
                    slot = 0;
                    b_hi = b_first;
                }
                if (++t == kTStages) {
                    t = 0;
                    phase ^= 1u;
                }
                buf ^= 1u;
            }
        }
        if (!ok)
            give_up(ERR_MMA_WAIT);
        __syncwarp();
    } else if (warp >= 2 + kEpilogueWarps) {
        // ---------------- converters: fp32 A tile -> hi and lo planes in tensor memory ----------------
        // A warp takes 32 pixels and half of a segment's 64 elements, one row of A. Every wait is for a
        // phase after one that the warp has seen (a parity cannot tell a phase from the one two before
        // it): a ring slot always holds rows of the same half, since the depth is even.
        const int half = (warp - 2 - kEpilogueWarps) >> 2;
        const int q = warp & 3;
        const int row = q * 32 + lane;
        const int swz = row & 7;  // 16-byte unit u of row r sits at unit u ^ (r & 7) of its row
        const int total = my_tiles * p.segs;
        const uint32_t a_full_a = smem_u32(a_full), a_empty_a = smem_u32(a_empty);
        int s = half, t = 0, g = 0;
        uint32_t a_phase = 0, t_phase = 1;
        bool ok = true;
        // Operands that the planes do not hold put the tile off
        uint32_t ordinal = 0;
        int m = 0, column = 0;
        bool strict = false, fits = true;
        LargestValues values;
        auto begin_tile = [&] {
            const int tile = first_tile + (int)ordinal * tile_step;
            const int tile_m = p.n_tiles == 1 ? tile : tile / p.n_tiles;
            m = tile_m * kBM + row;
            column = tile - tile_m * p.n_tiles;
            strict = __any_sync(0xffffffffu, columns->is_strict(column));
            fits = true;
            values.reset();
        };
        begin_tile();
        // (after a wait that ran out a warp goes on without waits and work: the two warps of a pixel quarter
        // meet at a barrier in every segment)
        for (int turn = 0; turn < total; ++turn) {
            float x[32];
            ok = ok && mbar_wait_u32(a_full_a + 8 * s, a_phase, abort_flag);
            ok = ok && mbar_wait_u32(done_a + 8 * t, t_phase, abort_flag);  // the segment four ago
            ok = __all_sync(0xffffffffu, ok);
            const bool there = ok && g * 2 + half < p.k_iters;
            const float4* src = reinterpret_cast<const float4*>(ring_a + s * kABytes + row * (kChans * 4));
#pragma unroll
            for (int u = 0; u < kChans / 4; ++u) {
                const float4 v = there ? src[u ^ swz] : make_float4(0.f, 0.f, 0.f, 0.f);
                x[4 * u + 0] = v.x;
                x[4 * u + 1] = v.y;
                x[4 * u + 2] = v.z;
                x[4 * u + 3] = v.w;
            }
            // the pixel's largest value, over both halves
            float m4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                m4[i] = fabsf(x[i]);
#pragma unroll
                for (int k = 4 + i; k < 32; k += 4)
                    m4[i] = fmaxf(m4[i], fabsf(x[k]));
            }
            float most = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
            float* exchange = half_most + (turn & 1) * 2 * kBM + row;
            exchange[half * kBM] = most;
            asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
            most = fmaxf(most, exchange[(half ^ 1) * kBM]);
            const uint32_t field = scale_field(most);
            const SplitScale<true> scale(field);
            values.take(most);
            if (ok) {
                // (the sums of eight segments ago have been taken: the accumulators of six ago
                // were free before the MMAs of four ago, which have retired)
                if (half == 0)
                    pixel_factor[(turn & 7) * kBM + row] = field_to_float(pixel_factor_field(field));
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ta = tmem_base + ((uint32_t)(q * 32) << 16) + kAccCols +
                                    (uint32_t)(t * kTCols + half * 16);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t hi[8], lo[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        split_f16(x[16 * h + 2 * i], x[16 * h + 2 * i + 1], scale, hi[i], lo[i]);
                    tmem_st8(ta + 8 * h, hi);
                    tmem_st8(ta + kTCols / 2 + 8 * h, lo);
                }
                if (strict && there) {
                    // (read again: kept for this, the values slowed the loop down for everyone, 2048^3 71 -> 78 us)
                    uint32_t least = 0xffffffffu;
#pragma unroll
                    for (int u = 0; u < kChans / 4; ++u) {
                        const float4 v = src[u ^ swz];
                        least = min(min(least, min(magnitude_0_last(v.x), magnitude_0_last(v.y))),
                                    min(magnitude_0_last(v.z), magnitude_0_last(v.w)));
                    }
                    fits = fits && least >= least_magnitude(field);
                    strict = __any_sync(0xffffffffu, columns->is_strict(column));  // (it may just have been found out)
                }
                // (a row behind the last pixel may hold whatever lies behind the input)
                if (g + 1 == p.segs)
                    put_tile_off_if(!(fits && values.fit()) && m < p.m_total, late_a, ordinal);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_u32(ready_a + 8 * t);
                    // The raw row goes back only now, when its values have been used: a load still
                    // on its way to a register is not ordered before the TMA's next write.
                    mbar_arrive_u32(a_empty_a + 8 * s);
                }
            }
            if (++g == p.segs) {
                g = 0;
                ++ordinal;
                begin_tile();
            }
            s += 2;
            if (s >= p.a_stages) {
                s -= p.a_stages;
                a_phase ^= 1u;
            }
            if (++t == kTStages) {
                t = 0;
                t_phase ^= 1u;
            }
        }
        if (!ok)
            give_up(ERR_PRODUCER_WAIT);
        __syncwarp();
    } else {
        // ---------------- epilogue: warps 2..9, TMEM lanes 32 * (warp % 4) .. ----------------
        const int q = warp & 3;
        const int row = q * 32 + lane;
        const int half = (warp - 2) >> 2;
        constexpr int kCols = kBN / 2;       // columns of this warp
        float* bias_row = reinterpret_cast<float*>(smem + kBiasOff) + (warp - 2) * 2 * kCols;
        float* factor_row = bias_row + kCols;
        const uint32_t turned_w = smem_u32(smem + kTurnOff) + (warp - 2) * (32 * kTurn * 4);
        uint32_t turn = 0;
        bool ok = true;
        if (lane == 0) {  // the accumulators of the first two segments are free
            mbar_arrive(&ready[0]);
            mbar_arrive(&ready[1]);
        }
        pdl_wait();  // before the first read of z and the first store
        find_column_states<32 * kEpilogueWarps, 5>(p.factor, p.oc, kBN, (int)threadIdx.x - 64, columns, &late->any);
        for (int tile = first_tile; tile < total_tiles && ok; tile += tile_step) {
            const int tile_n = tile % p.n_tiles, tile_m = tile / p.n_tiles;
            const int m = tile_m * kBM + row, n0 = tile_n * kBN;
            if (p.n_tiles > 1 || tile == first_tile) {  // once, where one column covers the channels
                __syncwarp();
#pragma unroll
                for (int j = lane; j < kCols; j += 32) {
                    const int ch = n0 + half * kCols + j;
                    bias_row[j] = p.ep.bias && ch < p.oc ? __ldg(p.ep.bias + ch) : 0.f;
                    factor_row[j] = ch < p.oc ? channel_factor(__float_as_uint(__ldg(p.factor + ch))) : 0.f;
                }
                __syncwarp();
            }
            if (p.ep.z && m < p.m_total) {
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
            const uint32_t lane_base =
                    tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * kCols);
            for (int g = 0; g < p.segs && ok; ++g, ++turn) {
                ok = mbar_wait(&done[turn % kTStages], (turn / kTStages) & 1u, abort_flag);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) {
                    give_up(ERR_EPILOGUE_WAIT);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const float f = pixel_factor[(turn & 7) * kBM + row];
                // (Each load is waited for in the statement that issues it: with a load in flight
                // across other code, a register that it has yet to write must never be spilled, and
                // with this many sums nothing guarantees that.)
#pragma unroll
                for (int c = 0; c < kCols / 16; ++c) {
                    uint32_t v[16];
                    tmem_ld16(lane_base + (turn & 1) * kBN + (uint32_t)(16 * c), v);
#pragma unroll
                    for (int j = 0; j < 16; ++j)
                        sum[16 * c + j] = __fmaf_rn(__uint_as_float(v[j]), f, sum[16 * c + j]);
                }
                // the warp's accumulators are in registers: hand the set back
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0)
                    mbar_arrive(&ready[(turn + 2) % kTStages]);
            }
            if (!ok)
                break;
            if (n0 + half * kCols < p.oc) {
                const F32RowsInLine rows{(size_t)(m - lane), (size_t)p.m_total};
                store_f32_rows<kCols, kTurn, true>(sum, p.ep, turned_w, factor_row, bias_row, rows,
                                                   n0 + half * kCols);
            }
        }
    }

    // ---------------- the tiles put off, teardown ----------------
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*(volatile uint32_t*)&late->any != 0 && !*abort_flag) {
        exact_tiles<kBN>(p, late, columns, tiles_b, tmem_base, exact_bars, abort_flag);
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
                     "r"(512)
                     : "memory");
    }
}

}  // namespace

// floats of the planes and factors of a filter [OC][taps][padded IC]
size_t conv_f32_half_filter_floats(const ConvF32Args& a) {
    return (size_t)a.oc * a.kh * a.kw * conv_f32_padded_ic(a.ic) + (size_t)(a.oc + 3) / 4 * 4;
}

int launch_conv_f32_pack_filter_half(
        const ConvF32Args& a, const float* flt_oihw, float* out, cudaStream_t st) {
    pack_filter_half_kernel<<<a.oc, 256, 0, st>>>(flt_oihw, out, a.oc, a.ic, conv_f32_padded_ic(a.ic),
                                                  a.kh, a.kw);
    return check_launch("pack_filter_f32_half");
}

int launch_matmul_f32_pack_half(int k, int n, const float* b, float* out, cudaStream_t st) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((n + 31) / 32 * kPackParts));
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kPackParts;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaLaunchKernelEx(&cfg, pack_matrix_half_kernel, b, out, k, n, conv_f32_padded_ic(k)) != cudaSuccess)
        return check_launch("pack_matrix_half");
    return check_launch("pack_matrix_half");
}

// map_a: rows of 32 channels and 128 pixels, as for conv_f32.cu. `weights`: the filter's tf32 planes, or the
// second operand of a matrix product as it is ([K][N])
int launch_conv_f32_half(
        const ConvF32Args& a, const CUtensorMap& map_a, bool a_tiled, const float* src, const float* planes,
        const float* weights, bool weights_raw, const float* bias, const float* z, float* dst, cudaStream_t st) {
    static KernelReady ready;
    if (!ready.smem(conv_f32_half_kernel, kDynamic))
        return check_launch("conv_f32_half smem attribute");
    const int icp = conv_f32_padded_ic(a.ic), taps = a.kh * a.kw;
    const cuuint64_t k_total = (cuuint64_t)taps * icp;
    CUtensorMap map_b;
    cuuint64_t dims[2] = {k_total, (cuuint64_t)2 * a.oc};
    cuuint64_t strides[1] = {k_total * 2};
    cuuint32_t box[2] = {(cuuint32_t)kSegK, (cuuint32_t)kBN};
    cuuint32_t estr[2] = {1, 1};
    const CUresult r = driver_api().tiled(
            &map_b, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)planes, dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
            CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return set_error(ST_RUNTIME, "cuTensorMapEncodeTiled(f32 filter planes) failed: %d", (int)r);
    HalfConvParams p;
    p.m_total = a.m;
    p.oc = a.oc;
    p.oh = a.oh;
    p.ow = a.ow;
    p.cblocks = icp / kChans;
    p.taps_w = a.kw;
    p.k_iters = taps * p.cblocks;
    p.segs = (p.k_iters + 1) / 2;
    p.sh = a.sh;
    p.sw = a.sw;
    p.base_h = -a.ph;
    p.base_w = -a.pw;
    p.m_tiles = (a.m + kBM - 1) / kBM;
    p.n_tiles = (a.oc + kBN - 1) / kBN;
    p.a_tiled = a_tiled ? 1 : 0;
    // the filter stays in shared memory where one tile column covers the channels and it leaves four rows
    // of A their place; else its segments go through a ring beside that of the rows
    const long long b_all = (long long)p.segs * kBBytes;
    p.b_resident = p.n_tiles == 1 && p.m_tiles > sm_count() && b_all + 4 * kABytes <= kTileBudget;
    p.b_stages = 3;
    const long long rest = kTileBudget - (p.b_resident ? b_all : (long long)p.b_stages * kBBytes);
    const int rows = (int)(rest / kABytes) / 2 * 2;
    p.a_stages = rows > kMaxAStages ? kMaxAStages : rows;
    p.ep.oc = a.oc;
    p.ep.act = a.act;
    p.ep.bias = bias;
    p.ep.z = z;
    p.ep.z_pitch = a.z_pitch;
    p.ep.dst = dst;
    p.ep.dst_pitch = a.dst_pitch;
    p.factor = planes + (size_t)a.oc * k_total;
    p.exact = conv_f32_exact_operands(a, src, weights, weights_raw);
    p.status = device_status_word(st);
    if (!p.status)
        return ST_MALLOC;
    const int total = p.m_tiles * p.n_tiles;
    const int grid = total < sm_count() ? total : sm_count();
    if (tuning().debug)
        fprintf(stderr, "conv_f32_half: grid %d tiles %d segments %d rings %d %d resident %d\n", grid, total,
                p.segs, p.a_stages, p.b_stages, p.b_resident);
    launch_pdl(Writes{dst, (size_t)a.m * a.dst_pitch * 4}, conv_f32_half_kernel, dim3(grid), dim3(kThreads),
               (size_t)kDynamic, st, map_a, map_b, p);
    return check_launch("conv_f32_half");
}

}  // namespace mb200
