// The kernel of conv_umma.cu and its launchers, compiled in one file per tile width (conv_umma_64.cu,
// _128.cu, _256.cu): all of them in one take the compiler four minutes.
#pragma once
#include <stdio.h>
#include <stdlib.h>

#include "conv_epilogue.cuh"
#include "internal.h"
#include "pdl.h"
#include "tuning.h"
#include "umma_ptx.cuh"

namespace mb200 {

using namespace umma;

namespace umma_conv {

constexpr int kBM = 128;     // output pixels per tile (UMMA M)
constexpr int kBK = 64;      // K bytes per pipeline stage of the 64-byte geometries
constexpr int kUmmaK = 32;   // K per tcgen05.mma kind::i8
constexpr int kStages = 6;         // most stages any variant uses (sizes the barrier arrays)
enum Geometry : int { GEOM_WIDE = 0, GEOM_TAP16 = 1, GEOM_WIDE128 = 2 };

// Per output-channel tile width. BN = 64 / 128: two accumulator buffers of BN columns, up
// to three CTAs per SM, two epilogue warps per TMEM lane quarter. BN = 256 (only with
// 128-byte rows): the two buffers fill the SM's 512 TMEM columns, so one CTA per SM, which
// then gets four epilogue warps per lane quarter and a larger register budget. The wide
// tile exists because the operands come from L2 at well under 100 bytes per clock and SM:
// a 128 x 128 tile needs 32 KB per 256 MMA cycles, a 128 x 256 tile 48 KB per 512.
template <int BN>
struct Shape {
    static constexpr int kEpilogueWarps = BN == 256 ? 16 : 8;
    static constexpr int kEpilogueThreads = 32 * kEpilogueWarps;
    static constexpr int kThreads = 64 + kEpilogueThreads;
    static constexpr int kMinCtas = BN == 256 ? 1 : 2;
};

// K bytes and pipeline depth per geometry. WIDE128 moves 128-channel rows (128-byte swizzle):
// half as many TMA requests and barrier round trips per byte as WIDE.
template <int BN, int GEOM>
struct Geom {
    static constexpr int kBKg = GEOM == GEOM_WIDE128 ? 128 : 64;
    static constexpr int kStagesG = GEOM == GEOM_WIDE128 ? (BN == 256 ? 4 : 3) : kStages;
};

struct UmmaConvParams {
    int m_total, oc, oh, ow;
    int cblocks;        // channel blocks per tap; the last may reach past the tap's channels
    int tap_step;       // filter bytes from a tap's last block to the next tap's first (kBKg, less the overhang)
    int taps_w;         // filter taps along W (TAP16: taps of the space-to-depth filter)
    int k_iters;        // pipeline stages per tile
    int sh, sw;         // output -> base pixel scaling
    int base_h, base_w; // coordinate of output (0,0)'s first tap (= -pad)
    int dh, dw;
    int m_tiles, n_tiles;
    int a_tiled;        // 1x1, stride 1, no padding: A is the plain matrix [pixels][channels]
    EpilogueParams ep;
    int8_t* dst;
    int* status;
    // cycles a bounded wait may take (kWaitCycles unless a self-test shortens it), and the
    // pipeline step of every tile that the producer leaves out (-1: none; self-test only)
    long long wait_cycles;
    int skip_step;
    // split-K (SPLITK kernels only): work items below `full_tiles` are whole tiles, the
    // tiles after them are cut into `split` parts of `k_per_part` pipeline steps each
    int full_tiles, split, k_per_part, total_items;
    // K split over a cluster (whole kernels without SPLITK): CTAs that share a tile's K loop, 1: none
    int csplit;
    int4* slabs;          // [split item][chunk][16-byte group][row]: one part's accumulators
    unsigned* counters;   // [split tile] parts finished; zero between launches
};

// One unit of work of a persistent CTA: a whole tile, or one K range of a split tile.
struct WorkItem {
    int tile, k0, k1;
    int slot;  // index of the split item (its slab), -1 for a whole tile
};

template <bool SPLITK>
__device__ __forceinline__ WorkItem decode_item(const UmmaConvParams& p, int item, int rank) {
    WorkItem w;
    if (!SPLITK && p.csplit > 1) {
        w.tile = item;
        w.k0 = p.k_iters * rank / p.csplit;
        w.k1 = p.k_iters * (rank + 1) / p.csplit;
        w.slot = -1;
    } else if (!SPLITK || item < p.full_tiles) {
        w.tile = item;
        w.k0 = 0;
        w.k1 = p.k_iters;
        w.slot = -1;
    } else {
        const int idx = item - p.full_tiles;
        const int t = idx / p.split, part = idx - t * p.split;
        w.tile = p.full_tiles + t;
        w.k0 = part * p.k_per_part;
        w.k1 = min(w.k0 + p.k_per_part, p.k_iters);
        w.slot = idx;
    }
    return w;
}

template <int BN, int GEOM>
struct SmemLayout {
    static constexpr int kABytes = kBM * Geom<BN, GEOM>::kBKg;
    static constexpr int kBBytes = BN * Geom<BN, GEOM>::kBKg;
    static constexpr int kTiles = Geom<BN, GEOM>::kStagesG * (kABytes + kBBytes);
    // after the tiles: full[kStages], empty[kStages], acc_full[2], acc_empty[2], drain,
    // the epilogue's own rendezvous (split-K), then three words
    static constexpr int kBarOff = kTiles;
    static constexpr int kTotal = kBarOff + (2 * kStages + 6) * 8 + 16;
    static constexpr int kDynamic = kTotal + 1024;  // room to align the tiles to 1024 bytes
};

template <int BN, int GEOM, bool SPLITK = false, int FORM = FORM_ANY>
__global__ void __launch_bounds__(Shape<BN>::kThreads, Shape<BN>::kMinCtas) conv_umma_kernel(
        const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
        const UmmaConvParams p) {
    using L = SmemLayout<BN, GEOM>;
    constexpr int kBKc = Geom<BN, GEOM>::kBKg;
    constexpr int kSt = Geom<BN, GEOM>::kStagesG;
    constexpr int kEpilogueWarps = Shape<BN>::kEpilogueWarps;
    constexpr int kPartPitch = BN + 4;  // int32 per row of a split tile's share
    static_assert(SPLITK || BN == 256 || kBM * kPartPitch * 4 <= L::kTiles, "the share takes the stages' place");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* tiles_a = smem;
    uint8_t* tiles_b = smem + kSt * L::kABytes;
    uint64_t* full_bar = (uint64_t*)(smem + L::kBarOff);
    uint64_t* empty_bar = full_bar + kStages;
    uint64_t* acc_full = empty_bar + kStages;  // [2]
    uint64_t* acc_empty = acc_full + 2;        // [2]
    uint64_t* drain_bar = acc_empty + 2;
    uint64_t* ep_bar = drain_bar + 1;
    uint32_t* tmem_slot = (uint32_t*)(ep_bar + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    volatile int* last_flag = (volatile int*)(tmem_slot + 2);

    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    const int total_tiles = SPLITK ? p.total_items : p.m_tiles * p.n_tiles;
    // split over a cluster: one tile per cluster, a K range per CTA
    const int rank = !SPLITK && p.csplit > 1 ? (int)cluster_rank() : 0;
    const int first_item = SPLITK ? (int)blockIdx.x : (int)blockIdx.x / p.csplit;
    const int item_step = !SPLITK && p.csplit > 1 ? total_tiles : (int)gridDim.x;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 32 * kEpilogueWarps);  // every epilogue thread arrives
        }
        mbar_init(drain_bar, 1);
        mbar_init(ep_bar, 32 * kEpilogueWarps);
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
                "r"(2 * BN)
                : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            // this thread runs alone in its warp and every instruction costs it several
            // cycles: stage, phase and filter tap are running counters, no division per step
            int s = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int item = first_item; item < total_tiles && ok; item += item_step) {
                const WorkItem w = decode_item<SPLITK>(p, item, rank);
                const int tile = w.tile;
                const int tile_n = tile % p.n_tiles, tile_m = tile / p.n_tiles;
                const int m0 = tile_m * kBM, n0 = tile_n * BN;
                const int img = m0 / (p.oh * p.ow);
                const int rem = m0 - img * (p.oh * p.ow);
                const int oy = rem / p.ow, ox = rem - oy * p.ow;
                const int base_w = ox * p.sw + p.base_w, base_h = oy * p.sh + p.base_h;
                int cb = 0, fx = 0, fy = 0, bx = 0;
                if (w.k0 != 0) {
                    // a later part of a split tile starts in the middle of the filter
                    cb = w.k0 % p.cblocks;
                    const int tap = w.k0 / p.cblocks;
                    fy = tap / p.taps_w;
                    fx = tap - fy * p.taps_w;
                    bx = tap * ((p.cblocks - 1) * kBKc + p.tap_step) + cb * kBKc;
                }
                if (item == first_item) {
                    pdl_wait();     // (the first tile is worked out before the wait)
                    pdl_release();  // the next kernel may take the SMs this one leaves free
                }
                for (int it = w.k0; it < w.k1; ++it) {
                    if (!mbar_wait(&empty_bar[s], phase ^ 1u, abort_flag, p.wait_cycles)) {
                        if (!*abort_flag) {
                            *abort_flag = 1;
                            atomicExch(p.status, ERR_PRODUCER_WAIT);
                        }
                        ok = false;
                        break;
                    }
                    if (it == p.skip_step) {
                        // self-test of the bounded waits: this stage is never filled (neither
                        // the byte count is announced nor a load issued), so the MMA thread's
                        // wait for it runs out and the kernel takes its give-up path
                        if (++s == kSt) {
                            s = 0;
                            phase ^= 1u;
                        }
                        continue;
                    }
                    mbar_expect_tx(&full_bar[s], (uint32_t)(L::kABytes + L::kBBytes));
                    uint8_t* sa = tiles_a + s * L::kABytes;
                    uint8_t* sb = tiles_b + s * L::kBBytes;
                    if (GEOM != GEOM_TAP16) {
                        if (p.a_tiled)
                            tma_load_2d(sa, &map_a, &full_bar[s], cb * kBKc, m0);
                        else
                            tma_load_im2col_4d(sa, &map_a, &full_bar[s], cb * kBKc, base_w, base_h,
                                               img, (uint16_t)(fx * p.dw), (uint16_t)(fy * p.dh));
                        // (an overhanging block reads the next tap's filter bytes, or zeros behind the
                        // last: its activation bytes are zeros)
                        tma_load_2d(sb, &map_b, &full_bar[s], bx, n0);
                        bx += kBKc;
                        if (++cb == p.cblocks) {
                            cb = 0;
                            bx += p.tap_step - kBKc;
                            if (++fx == p.taps_w) {
                                fx = 0;
                                ++fy;
                            }
                        }
                    } else {
#pragma unroll
                        for (int t = 0; t < 4; ++t) {
                            tma_load_im2col_4d(sa + t * (kBM * 16), &map_a, &full_bar[s], 0, base_w,
                                               base_h, img, (uint16_t)fx, (uint16_t)fy);
                            tma_load_2d(sb + t * (BN * 16), &map_b, &full_bar[s], (it * 4 + t) * 16,
                                        n0);
                            if (++fx == p.taps_w) {
                                fx = 0;
                                ++fy;
                            }
                        }
                    }
                    if (++s == kSt) {
                        s = 0;
                        phase ^= 1u;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer (the whole warp waits, one lane issues) ----------------
        // Instructions between two MMAs show as idle tensor time: descriptor words are running
        // sums, every lane takes the loop so that they stay in uniform registers.
        const uint32_t leader = elect_one() ? 1u : 0u;
        constexpr uint32_t idesc = umma_idesc_s8(kBM, BN);
        // one descriptor per operand and stage; a K step only moves the address field (16-byte
        // units): +32 bytes inside the swizzled row, or two 16-byte tap blocks in the plain
        // layout. 128-byte swizzle: 8-row groups 1024 bytes apart; 64-byte: 512.
        const uint64_t a0 = GEOM == GEOM_WIDE128 ? umma_smem_desc(smem_u32(tiles_a), 16, 1024, 2)
                            : GEOM == GEOM_WIDE  ? umma_smem_desc(smem_u32(tiles_a), 16, 512, 4)
                                                 : umma_smem_desc(smem_u32(tiles_a), kBM * 16, 128, 0);
        const uint64_t b0 = GEOM == GEOM_WIDE128 ? umma_smem_desc(smem_u32(tiles_b), 16, 1024, 2)
                            : GEOM == GEOM_WIDE  ? umma_smem_desc(smem_u32(tiles_b), 16, 512, 4)
                                                 : umma_smem_desc(smem_u32(tiles_b), BN * 16, 128, 0);
        constexpr uint32_t a_k = GEOM == GEOM_TAP16 ? 2 * (kBM * 16) / 16 : 32 / 16;
        constexpr uint32_t b_k = GEOM == GEOM_TAP16 ? 2 * (BN * 16) / 16 : 32 / 16;
        const uint32_t a_hi = (uint32_t)(a0 >> 32), b_hi = (uint32_t)(b0 >> 32);
        const uint32_t full_a = smem_u32(full_bar), empty_a = smem_u32(empty_bar);
        const uint32_t acc_full_a = smem_u32(acc_full), acc_empty_a = smem_u32(acc_empty);
        uint32_t a_lo = (uint32_t)a0, b_lo = (uint32_t)b0;
        uint32_t phase = 0, buf = 0, acc_parity = 1;
        int s = 0;
        bool ok = true;
        for (int item = first_item; item < total_tiles && ok; item += item_step) {
            const WorkItem w = decode_item<SPLITK>(p, item, rank);
            // the epilogue must have drained this accumulator buffer
            ok = mbar_wait_u32(acc_empty_a + 8 * buf, acc_parity, abort_flag, p.wait_cycles);
            if (!ok) {
                if (!*abort_flag) {
                    *abort_flag = 1;
                    atomicExch(p.status, ERR_MMA_ACC_WAIT);
                }
                break;
            }
            const uint32_t tmem_d = tmem_base + buf * BN;
            uint32_t acc = 0;
            for (int it = w.k0; it < w.k1; ++it) {
                ok = mbar_wait_u32(full_a + 8 * s, phase, abort_flag, p.wait_cycles);
                if (!ok) {
                    if (!*abort_flag) {
                        *abort_flag = 1;
                        atomicExch(p.status, ERR_MMA_WAIT);
                    }
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                umma_s8(leader, tmem_d, a_lo, a_hi, b_lo, b_hi, idesc, acc);
#pragma unroll
                for (int k = 1; k < kBKc / kUmmaK; ++k)
                    umma_s8(leader, tmem_d, a_lo + k * a_k, a_hi, b_lo + k * b_k, b_hi, idesc, 1);
                umma_commit_if(leader, empty_a + 8 * s);  // frees the stage once these retire
                acc = 1;
                a_lo += L::kABytes / 16;
                b_lo += L::kBBytes / 16;
                if (++s == kSt) {
                    s = 0;
                    phase ^= 1u;
                    a_lo = (uint32_t)a0;
                    b_lo = (uint32_t)b0;
                }
            }
            if (!ok)
                break;
            umma_commit_if(leader, acc_full_a + 8 * buf);
            buf ^= 1u;
            acc_parity ^= buf ^ 1u;  // flips each time buffer 0 comes round again
        }
        __syncwarp();
    } else {
        // ---------------- epilogue: warps 2..9, TMEM lanes 32*(warp%4).. ----------------
        const int q = warp & 3;
        const int row = q * 32 + lane;
        int local = 0;
        bool ok = true;
        uint32_t ep_phase = 0;  // parity of the epilogue's own rendezvous (split-K)
        pdl_wait();  // before the first read of z and the first store
        const bool unbounded = form_is_chain(FORM) && chain_unbounded(p.ep);
        uint32_t asked = 0;
        if (!SPLITK && p.csplit <= 1 && first_item < total_tiles) {
            // the first tile's parameters and residual come while its MMAs run
            const int n0 = first_item % p.n_tiles * BN, m = first_item / p.n_tiles * kBM + row;
            const int ch0 = n0 + ((warp - 2) >> 2) * (BN / (kEpilogueWarps / 4));
            asked = ask_for_params(p.ep, ch0, BN / (kEpilogueWarps / 4), m < p.m_total, (size_t)m * p.oc + ch0);
        }
        for (int item = first_item; item < total_tiles && ok; item += item_step, ++local) {
            const WorkItem w = decode_item<SPLITK>(p, item, rank);
            const int tile = w.tile;
            const int buf = local & 1;
            const uint32_t acc_phase = (uint32_t)(local >> 1) & 1u;
            const int tile_n = tile % p.n_tiles, tile_m = tile / p.n_tiles;
            const int m = tile_m * kBM + row, n0 = tile_n * BN;
            ok = mbar_wait(&acc_full[buf], acc_phase, abort_flag, p.wait_cycles);
            if (!ok && !*abort_flag) {
                *abort_flag = 1;
                atomicExch(p.status, ERR_EPILOGUE_WAIT);
            }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok)
                break;
            keep(asked);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN);
            const int half = (warp - 2) >> 2;
            // each warp takes a run of adjacent chunks: its thread's bytes are contiguous
            constexpr int kChunksPerWarp = (BN / 32) / (kEpilogueWarps / 4);
            static_assert(kChunksPerWarp >= 1, "every epilogue warp must own a chunk");
            if (SPLITK && w.slot >= 0) {
                // One K range of a split tile. Its raw accumulators go to this item's slab;
                // a slab is laid out [chunk][16-byte group][row], so a warp's 16-byte stores
                // (and the loads of the CTA that finishes the tile, whose threads own the same
                // rows and chunks) are 512 contiguous bytes. The CTA that finds the tile's
                // other parts already counted sums all slabs and requantises; nobody waits
                // for another CTA.
                constexpr int kSlabVecs = (BN / 32) * 8 * kBM;
                int4* slab = p.slabs + (size_t)w.slot * kSlabVecs;
#pragma unroll 1
                for (int c = half * kChunksPerWarp; c < (half + 1) * kChunksPerWarp; ++c) {
                    uint32_t v[32];
                    tmem_ld32(taddr + (uint32_t)(c * 32), v);
                    if (c + 1 == (half + 1) * kChunksPerWarp) {
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        mbar_arrive(&acc_empty[buf]);
                    }
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        __stcg(slab + (c * 8 + k) * kBM + row,
                               make_int4((int)v[4 * k], (int)v[4 * k + 1], (int)v[4 * k + 2],
                                         (int)v[4 * k + 3]));
                }
                __threadfence();  // the slab is visible device-wide before the part is counted
                mbar_arrive(ep_bar);
                ok = mbar_wait(ep_bar, ep_phase, abort_flag, p.wait_cycles);
                ep_phase ^= 1u;
                if (ok && threadIdx.x == 64) {
                    unsigned* counter = p.counters + (w.tile - p.full_tiles);
                    const unsigned before = atomicAdd(counter, 1u);
                    const bool last = before + 1u == (unsigned)p.split;
                    if (last)
                        *counter = 0;  // every part has been counted: ready for the next launch
                    *last_flag = last ? 1 : 0;
                }
                if (ok) {
                    mbar_arrive(ep_bar);
                    ok = mbar_wait(ep_bar, ep_phase, abort_flag, p.wait_cycles);
                    ep_phase ^= 1u;
                }
                if (!ok && !*abort_flag) {
                    *abort_flag = 1;
                    atomicExch(p.status, ERR_EPILOGUE_WAIT);
                }
                ok = __all_sync(0xffffffffu, ok);
                if (!ok)
                    break;
                if (*last_flag) {
                    __threadfence();
                    const int4* first = p.slabs + (size_t)(w.slot - w.slot % p.split) * kSlabVecs;
#pragma unroll 1
                    for (int c = half * kChunksPerWarp; c < (half + 1) * kChunksPerWarp; ++c) {
                        uint32_t v[32];
#pragma unroll
                        for (int j = 0; j < 32; ++j)
                            v[j] = 0;
                        for (int part = 0; part < p.split; ++part) {
                            const int4* s4 = first + (size_t)part * kSlabVecs + (c * 8) * kBM + row;
#pragma unroll
                            for (int k = 0; k < 8; ++k) {
                                const int4 t = __ldcg(s4 + k * kBM);
                                v[4 * k] += (uint32_t)t.x;
                                v[4 * k + 1] += (uint32_t)t.y;
                                v[4 * k + 2] += (uint32_t)t.z;
                                v[4 * k + 3] += (uint32_t)t.w;
                            }
                        }
                        const int ch0 = n0 + c * 32;
                        if (m < p.m_total && ch0 < p.oc)
                            epilogue_store<32>(v, p.ep, p.dst, (size_t)m * p.oc + ch0, ch0);
                    }
                }
                continue;
            }
            if (!SPLITK && p.csplit > 1) {
                // This CTA's share of the K loop: raw accumulators into shared memory in place
                // of the stages (every load has been consumed, every MMA has retired); the
                // cluster adds the shares up below.
                int4* part = reinterpret_cast<int4*>(smem + (size_t)row * (kPartPitch * 4));
#pragma unroll 1
                for (int c = half * kChunksPerWarp; c < (half + 1) * kChunksPerWarp; ++c) {
                    uint32_t v[32];
                    tmem_ld32(taddr + (uint32_t)(c * 32), v);
#pragma unroll
                    for (int k = 0; k < 8; ++k)
                        part[c * 8 + k] = make_int4((int)v[4 * k], (int)v[4 * k + 1],
                                                    (int)v[4 * k + 2], (int)v[4 * k + 3]);
                }
                continue;
            }
#pragma unroll 1
            for (int c = half * kChunksPerWarp; c < (half + 1) * kChunksPerWarp; ++c) {
                if constexpr (FORM != FORM_ANY) {
                    const int ch0 = n0 + c * 32;
                    uint64_t* release =
                            c + 1 == (half + 1) * kChunksPerWarp ? &acc_empty[buf] : nullptr;
                    if (ch0 < p.oc) {
                        epilogue_form_chunk<FORM>(taddr + (uint32_t)(c * 32), p.ep, p.dst,
                                                  (size_t)m * p.oc + ch0, ch0, m < p.m_total,
                                                  unbounded, release);
                    } else if (release) {
                        mbar_arrive(release);
                    }
                } else {
                    uint32_t v[32];
                    __syncwarp();
                    tmem_ld32(taddr + (uint32_t)(c * 32), v);
                    if (c + 1 == (half + 1) * kChunksPerWarp) {
                        // all of this thread's accumulators are in registers: hand the buffer back
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        mbar_arrive(&acc_empty[buf]);
                    }
                    const int ch0 = n0 + c * 32;
                    if (m < p.m_total && ch0 < p.oc)
                        epilogue_store<32>(v, p.ep, p.dst, (size_t)m * p.oc + ch0, ch0);
                }
            }
        }
    }

    if (!SPLITK && p.csplit > 1) {
        // Every CTA of the cluster comes here, whatever became of its waits; each finishes an
        // equal share of the rows. A thread's items lie 256 apart, in one channel quad: bias,
        // scales and residual are fetched while the shares arrive, and the CTA says that it
        // has read the others' shares before it stores (an arrival behind the stores waits for
        // them to be performed: 3 to 4.5 us from the last MMA to the end with everything
        // in line, on tiles of a batch of one).
        __syncwarp();
        cluster_arrive();
        constexpr int kQuads = BN / 4, kRowStep = 32 * kEpilogueWarps / kQuads;
        constexpr int kItems = kBM / 2 / kRowStep;  // at most (two CTAs)
        const int et = (int)threadIdx.x - 64;
        const int rows = kBM / p.csplit;
        const int tile_n = first_item % p.n_tiles, tile_m = first_item / p.n_tiles;
        const int c = (et & (kQuads - 1)) * 4, ch = tile_n * BN + c;
        const int r0 = rank * rows + et / kQuads;
        const int m0 = tile_m * kBM + r0;
        QuadParams qp;
        uint32_t zw[kItems];
        int v[kItems][4];
        int items = 0;
        if (et >= 0 && ch < p.oc) {
            qp = quad_params(p.ep, ch);
#pragma unroll
            for (int k = 0; k < kItems; ++k) {
                zw[k] = 0;
                if (et / kQuads + k * kRowStep < rows && m0 + k * kRowStep < p.m_total) {
                    items = k + 1;
                    zw[k] = quad_z(p.ep, (size_t)(m0 + k * kRowStep) * p.oc + ch, ch);
                }
            }
        }
        cluster_wait();  // the shares are in place
        if (*abort_flag)
            items = 0;
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            if (k < items) {
                const uint32_t at =
                        smem_u32(smem) + (uint32_t)(((r0 + k * kRowStep) * kPartPitch + c) * 4);
                uint4 x[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)  // all shares' loads in flight together
                    x[i] = i < p.csplit ? ld_cluster_v4(at, i) : make_uint4(0, 0, 0, 0);
                v[k][0] = v[k][1] = v[k][2] = v[k][3] = 0;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    v[k][0] += (int)x[i].x;
                    v[k][1] += (int)x[i].y;
                    v[k][2] += (int)x[i].z;
                    v[k][3] += (int)x[i].w;
                }
            }
        }
        __syncwarp();
        cluster_arrive();  // (a release: the loads above are done)
#pragma unroll
        for (int k = 0; k < kItems; ++k)
            if (k < items) {
                const size_t off = (size_t)(m0 + k * kRowStep) * p.oc + ch;
                if constexpr (FORM == FORM_NCHW)
                    nchw_quad(v[k], p.ep, qp, p.dst, off, ch);
                else
                    epilogue_quad(v[k], p.ep, qp, zw[k], p.dst, off, ch);
            }
        __syncwarp();
        cluster_wait();  // nobody leaves while its share may still be read
    }

    // ---------------- teardown ----------------
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag) {
        // a wait ran out: let loads in flight land and MMAs retire (both bounded) before
        // the shared memory and TMEM are given back
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
                     "r"(2 * BN)
                     : "memory");
    }
}

// ------------------------------------------------------------------------------------------
// host side: tensor maps and launch
// ------------------------------------------------------------------------------------------
template <int BN, int GEOM, bool SPLITK = false, int FORM = FORM_ANY>
bool umma_kernel_ready() {
    static KernelReady ready;
    return ready.smem(conv_umma_kernel<BN, GEOM, SPLITK, FORM>, SmemLayout<BN, GEOM>::kDynamic);
}

template <int BN, int GEOM, bool SPLITK = false, int FORM = FORM_ANY>
int launch_form(
        const CUtensorMap& ma, const CUtensorMap& mb, const UmmaConvParams& p, cudaStream_t st) {
    if (!umma_kernel_ready<BN, GEOM, SPLITK, FORM>())
        return check_launch("conv_umma smem attribute");
    // persistent CTAs: as many as the SM holds at once
    constexpr int kThreads = Shape<BN>::kThreads;
    static ResidentCtas resident;
    const int per_sm = resident.per_sm(conv_umma_kernel<BN, GEOM, SPLITK, FORM>, kThreads,
                                       SmemLayout<BN, GEOM>::kDynamic, 2 * BN);
    const int total = SPLITK ? p.total_items : p.m_tiles * p.n_tiles;
    int grid = sm_count() * per_sm;
    if (grid > total || p.csplit > 1)
        grid = total * p.csplit;
    if (tuning().debug)
        fprintf(stderr, "conv_umma<%d,%d,%d,%d>: csplit %d per_sm %d grid %d items %d (whole tiles %d, split %d) smem %d\n",
                BN, GEOM, (int)SPLITK, FORM, p.csplit, per_sm, grid, total, SPLITK ? p.full_tiles : total,
                SPLITK ? p.split : 1, SmemLayout<BN, GEOM>::kDynamic);
    const size_t outputs = (size_t)p.m_total * p.oc;
    const Writes writes = p.ep.acc_out ? Writes{p.ep.acc_out, outputs * 4} : Writes{p.dst, outputs};
    launch_pdl_cluster(writes, conv_umma_kernel<BN, GEOM, SPLITK, FORM>, dim3(grid), dim3(kThreads),
                       (size_t)SmemLayout<BN, GEOM>::kDynamic, p.csplit, st, ma, mb, p);
    return check_launch("conv_umma");
}

// the instantiation with the launch's epilogue (a split tile has its own, epilogue_quad)
template <int BN, int GEOM>
int launch_kernel(
        const CUtensorMap& ma, const CUtensorMap& mb, const UmmaConvParams& p, cudaStream_t st) {
    switch (p.ep.nchw_plane                              ? FORM_NCHW
            : p.csplit > 1 || !tuning().epilogue_forms ? FORM_ANY
                                                       : epilogue_form(p.ep, p.dst)) {
        case FORM_FMA_RELU: return launch_form<BN, GEOM, false, FORM_FMA_RELU>(ma, mb, p, st);
        case FORM_FMA_NONE: return launch_form<BN, GEOM, false, FORM_FMA_NONE>(ma, mb, p, st);
        case FORM_FMA_ADD_RELU: return launch_form<BN, GEOM, false, FORM_FMA_ADD_RELU>(ma, mb, p, st);
        case FORM_CHAIN_RELU: return launch_form<BN, GEOM, false, FORM_CHAIN_RELU>(ma, mb, p, st);
        case FORM_CHAIN_NONE: return launch_form<BN, GEOM, false, FORM_CHAIN_NONE>(ma, mb, p, st);
        case FORM_CHAIN_ADD_RELU:
            return launch_form<BN, GEOM, false, FORM_CHAIN_ADD_RELU>(ma, mb, p, st);
        case FORM_FMA_RAGGED: return launch_form<BN, GEOM, false, FORM_FMA_RAGGED>(ma, mb, p, st);
        case FORM_CHAIN_RAGGED: return launch_form<BN, GEOM, false, FORM_CHAIN_RAGGED>(ma, mb, p, st);
        case FORM_NCHW: return launch_form<BN, GEOM, false, FORM_NCHW>(ma, mb, p, st);
        default: return launch_form<BN, GEOM>(ma, mb, p, st);
    }
}

template <int BN, int GEOM>
int umma_clusters(int size) {
    static ClusterCapacity capacity;
    if (!umma_kernel_ready<BN, GEOM>())
        return 0;
    return capacity.clusters(conv_umma_kernel<BN, GEOM>, size, Shape<BN>::kThreads,
                             SmemLayout<BN, GEOM>::kDynamic);
}

}  // namespace umma_conv
}  // namespace mb200
