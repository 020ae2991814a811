// qint8 ConvBias / matrix product on the tensor cores with operands fetched by ordinary loads.
//
// The TMA kernels (conv_umma.cu, conv_patch.cu) want rows that start on 16-byte boundaries, NHWC and
// tensor maps over at least 128 KiB. What they leave out came down to one CUDA thread per output
// value (conv_direct_kernel): a 1113 x 983 x 1535 product took 2630 us, 24 here; 24 -> 256 channels 3x3
// over 10 x 31 x 104 538 and 45. Here the same implicit GEMM (128
// output pixels x 64 channels per tile, tcgen05.mma kind::i8, int32 accumulators in tensor memory)
// gets its operands from eight loader warps that write them in the swizzled K-major layout the MMAs
// read:
//
//   GATHER_VEC16  NHWC, channels % 16 == 0: 16 bytes of one filter tap per load
//   GATHER_WORDS  NHWC, channels % 4 == 0: four bytes per load
//   GATHER_ROWS   1x1 filter, stride 1: contiguous rows of any length and alignment, aligned words
//                 shifted into place
//   GATHER_NCHW   the reference's own layouts, NCHW source, OIHW filter and NCHW result, for a short K:
//                 a byte per load (32 consecutive pixels per warp). K runs channel by channel and tap
//                 by tap inside, as the filter lies in memory, so nothing is re-laid: one launch
//                 instead of three
//
// K runs in the filter's memory order in every form, so the filter rows are contiguous and are
// fetched like GATHER_ROWS. Each thread has the loads of one 64-byte step in flight while it writes
// the step before; with three CTAs per SM that hides most of their latency. One tile per CTA.
//
// Replaces the loop nest of compiler/lib/KernelGen/BareMetal/ConvKernel.cpp:305-344.
#include <stdio.h>

#include "conv_epilogue.cuh"
#include "internal.h"
#include "pdl.h"
#include "tuning.h"
#include "umma_ptx.cuh"

namespace mb200 {

using namespace umma;

namespace {

constexpr int kBM = 128, kBN = 64, kBK = 64;
constexpr int kStages = 4;
constexpr int kLoaders = 256;
constexpr int kThreads = kLoaders + 32;
constexpr int kABytes = kBM * kBK, kBBytes = kBN * kBK;
constexpr int kMaxTaps = 49;
constexpr int kSmem = kStages * (kABytes + kBBytes) + 1024;

enum GatherMode : int { GATHER_VEC16 = 0, GATHER_WORDS = 1, GATHER_ROWS = 2, GATHER_NCHW = 3 };

struct GatherParams {
    const int8_t *src, *flt;
    size_t src_bytes, flt_bytes;
    int m_total, oc, k_total;
    int ic, ih, iw, oh, ow, kh, kw, sh, sw, ph, pw, dh, dw;
    int n_tiles;
    int src_vec, flt_vec;  // rows start on 16-byte boundaries and are a multiple of 16 bytes long
    EpilogueParams ep;
    int8_t* dst;
    int* status;
};

// 16 bytes of a row on their way: the aligned words they lie in. They are shifted into place only when
// they are written (place()), a step later: a use here would wait for the load.
struct RawUnit {
    uint32_t w[5];
};
// The unit at `p`, of which `count` bytes exist. No byte outside [lo, hi) is read.
__device__ __forceinline__ RawUnit fetch_row(
        const int8_t* p, int count, bool vec, const int8_t* lo, const int8_t* hi) {
    RawUnit r;
#pragma unroll
    for (int i = 0; i < 5; ++i)
        r.w[i] = 0;
    if (count <= 0)
        return r;
    if (vec) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
        r.w[0] = v.x, r.w[1] = v.y, r.w[2] = v.z, r.w[3] = v.w;
        return r;
    }
    const int8_t* base = (const int8_t*)((uintptr_t)p & ~(uintptr_t)3);
    if (base >= lo && base + 20 <= hi) {
#pragma unroll
        for (int i = 0; i < 5; ++i)
            r.w[i] = __ldg(reinterpret_cast<const uint32_t*>(base) + i);
    } else {  // the tensor's ends, byte by byte (one behind the other their loads took 6 us)
        uint32_t v[20];
#pragma unroll
        for (int i = 0; i < 20; ++i) {
            const int8_t* at = base + i;
            const bool ok = at >= lo && at < hi;
            v[i] = (uint32_t)(uint8_t)__ldg(ok ? at : lo);
            v[i] = ok ? v[i] : 0u;
        }
#pragma unroll
        for (int i = 0; i < 5; ++i)
            r.w[i] = v[4 * i] | v[4 * i + 1] << 8 | v[4 * i + 2] << 16 | v[4 * i + 3] << 24;
    }
    return r;
}
// ... the 16 bytes themselves: `shift` bits into the words, `count` bytes of them, then zeros
__device__ __forceinline__ uint4 place(const RawUnit& raw, uint32_t shift, int count) {
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        r[i] = __funnelshift_r(raw.w[i], raw.w[i + 1], shift);
        const int left = count - 4 * i;
        if (left < 4)
            r[i] = left <= 0 ? 0u : r[i] & ((1u << (8 * left)) - 1u);
    }
    return make_uint4(r[0], r[1], r[2], r[3]);
}

// Where a thread's K position stands: filter tap and channel
struct TapPos {
    int c, fx, fy;
    __device__ __forceinline__ void carry(const GatherParams& p) {
        while (c >= p.ic) {
            c -= p.ic;
            if (++fx == p.kw) {
                fx = 0;
                ++fy;
            }
        }
    }
};

template <int MODE>
__global__ void __launch_bounds__(kThreads, 3) conv_gather_kernel(const GatherParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* tiles_a = smem;
    uint8_t* tiles_b = smem + kStages * kABytes;
    __shared__ uint64_t full_bar[kStages], empty_bar[kStages], acc_full, drain_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_word;
    __shared__ QuadParams side[kBN / 4];
    __shared__ int tap_off[kMaxTaps];
    volatile int* abort_flag = &abort_word;

    const int warp = uniform_warp_index(), lane = threadIdx.x & 31;
    const int tile_n = blockIdx.x % p.n_tiles, tile_m = blockIdx.x / p.n_tiles;
    const int m0 = tile_m * kBM, n0 = tile_n * kBN;
    const int steps = (p.k_total + kBK - 1) / kBK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full_bar[s], kLoaders / 32);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&acc_full, 1);
        mbar_init(&drain_bar, 1);
        abort_word = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (MODE == GATHER_NCHW && threadIdx.x < p.kh * p.kw) {
        const int fy = threadIdx.x / p.kw, fx = threadIdx.x - fy * p.kw;
        tap_off[threadIdx.x] = fy * p.dh * p.iw + fx * p.dw;
    }
    if (warp == kLoaders / 32) {
        asm volatile(
                "tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                        smem_u32(&tmem_slot)),
                "r"(kBN)
                : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_slot;

    if (warp < kLoaders / 32) {
        // ---------------- loaders, then epilogue ----------------
        pdl_wait();
        if (threadIdx.x == 0)
            pdl_release();
        if (threadIdx.x < kBN / 4)
            side[threadIdx.x] = quad_params(p.ep, n0 + 4 * (int)threadIdx.x);
        const int pixels = p.oh * p.ow;
        const int8_t *src_hi = p.src + p.src_bytes, *flt_hi = p.flt + p.flt_bytes;
        // Where a thread's two units of A lie in the step's tile. NHWC: four lanes have a pixel's 64
        // bytes, a thread the same unit of two pixels (with a pixel per lane every load of a warp touched
        // 32 lines: 1113 x 983 x 1535 took 43 us). NCHW: a pixel per lane, two units of it.
        constexpr bool kNchw = MODE == GATHER_NCHW;
        const int u = kNchw ? (int)(threadIdx.x >> 7) * 2 : (int)(threadIdx.x & 3);
        const int row0 = kNchw ? (int)threadIdx.x & (kBM - 1) : (int)threadIdx.x >> 2;
        const int row1 = kNchw ? row0 : row0 + 64, u1 = kNchw ? u + 1 : u;
        // B: the same four lanes per row
        const int b_row = threadIdx.x >> 2, b_u = threadIdx.x & 3;
        const bool b_in = n0 + b_row < p.oc;
        const int8_t* b_ptr = p.flt + (size_t)(b_in ? n0 + b_row : 0) * p.k_total + b_u * 16;
        int b_left = b_in ? p.k_total - b_u * 16 : 0;

        // a pixel's place: its image, the position of the first filter tap
        struct Pixel {
            const int8_t* image;
            int iy, ix;
            bool in;
        };
        auto pixel = [&](int row) {
            const int m = m0 + row;
            const bool in = m < p.m_total;
            const int img = m / pixels, rem = m - img * pixels;
            return Pixel{p.src + (size_t)(in ? img : 0) * p.ih * p.iw * p.ic, rem / p.ow * p.sh - p.ph,
                         rem % p.ow * p.sw - p.pw, in};
        };
        const Pixel px0 = pixel(row0), px1 = pixel(row1);
        TapPos at{u * 16, 0, 0};  // NHWC with a filter: running position of the thread's unit
        const int8_t *a_ptr0 = p.src, *a_ptr1 = p.src;
        int a_left0 = 0, a_left1 = 0, taps = 1, tap = 0, ch = 0;
        uint64_t tap_in = 0;  // NCHW: filter taps that lie inside the image
        if constexpr (MODE == GATHER_ROWS) {
            a_ptr0 = p.src + (size_t)(px0.in ? m0 + row0 : 0) * p.ic + u * 16;
            a_ptr1 = p.src + (size_t)(px1.in ? m0 + row1 : 0) * p.ic + u * 16;
            a_left0 = px0.in ? p.k_total - u * 16 : 0;
            a_left1 = px1.in ? p.k_total - u * 16 : 0;
        } else if constexpr (kNchw) {
            taps = p.kh * p.kw;
            if (px0.in) {
                for (int fy = 0, t = 0; fy < p.kh; ++fy)
                    for (int fx = 0; fx < p.kw; ++fx, ++t)
                        if ((unsigned)(px0.iy + fy * p.dh) < (unsigned)p.ih &&
                            (unsigned)(px0.ix + fx * p.dw) < (unsigned)p.iw)
                            tap_in |= 1ull << t;
            }
            ch = u * 16 / taps;
            tap = u * 16 - ch * taps;
        } else {
            at.carry(p);
        }

        // the 16 bytes of a pixel at position `t` (NHWC): all of one tap, or word by word
        auto unit_nhwc = [&](const Pixel& px, TapPos t) {
            uint32_t w[4] = {0, 0, 0, 0};
            if constexpr (MODE == GATHER_VEC16) {
                const int iy = px.iy + t.fy * p.dh, ix = px.ix + t.fx * p.dw;
                if (px.in && t.fy < p.kh && (unsigned)iy < (unsigned)p.ih && (unsigned)ix < (unsigned)p.iw)
                    return __ldg(reinterpret_cast<const uint4*>(
                            px.image + ((size_t)iy * p.iw + ix) * p.ic + t.c));
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int iy = px.iy + t.fy * p.dh, ix = px.ix + t.fx * p.dw;
                    if (px.in && t.fy < p.kh && (unsigned)iy < (unsigned)p.ih &&
                        (unsigned)ix < (unsigned)p.iw)
                        w[i] = __ldg(reinterpret_cast<const uint32_t*>(
                                px.image + ((size_t)iy * p.iw + ix) * p.ic + t.c));
                    t.c += 4;
                    t.carry(p);
                }
            }
            return make_uint4(w[0], w[1], w[2], w[3]);
        };
        // the 16 bytes from channel c, tap t on (NCHW)
        const long long plane = (long long)p.ih * p.iw;
        const long long corner = (long long)px0.iy * p.iw + px0.ix;
        auto unit_nchw = [&](int c, int t) {
            uint32_t w[4];
            long long base = c * plane + corner;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t b[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    // (no branch between the loads; what does not exist reads the image's first byte)
                    const bool ok = c < p.ic && ((tap_in >> t) & 1);
                    const long long off = ok ? base + tap_off[t] : 0;
                    b[j] = (uint32_t)(uint8_t)__ldg(px0.image + off);
                    b[j] = ok ? b[j] : 0u;
                    const bool wrap = ++t == taps;
                    t = wrap ? 0 : t;
                    c += wrap;
                    base += wrap ? plane : 0;
                }
                w[i] = pack4_prmt((int)b[0], (int)b[1], (int)b[2], (int)b[3]);
            }
            return make_uint4(w[0], w[1], w[2], w[3]);
        };
        // requests the step's units, and on to the next step
        struct Units {
            RawUnit a0, a1, b;
        };
        auto raw = [](uint4 v) { return RawUnit{{v.x, v.y, v.z, v.w, 0}}; };
        auto fetch = [&]() {
            Units v;
            if constexpr (MODE == GATHER_ROWS) {
                v.a0 = fetch_row(a_ptr0, a_left0, p.src_vec, p.src, src_hi);
                v.a1 = fetch_row(a_ptr1, a_left1, p.src_vec, p.src, src_hi);
                a_ptr0 += kBK;
                a_ptr1 += kBK;
                a_left0 -= kBK;
                a_left1 -= kBK;
            } else if constexpr (kNchw) {
                v.a0 = raw(unit_nchw(ch, tap));
                int t = tap + 16, c = ch;
                while (t >= taps)
                    t -= taps, ++c;
                v.a1 = raw(unit_nchw(c, t));
                tap += kBK;
                while (tap >= taps)
                    tap -= taps, ++ch;
            } else {
                v.a0 = raw(unit_nhwc(px0, at));
                v.a1 = raw(unit_nhwc(px1, at));
                at.c += kBK;
                at.carry(p);
            }
            v.b = fetch_row(b_ptr, b_left, p.flt_vec, p.flt, flt_hi);
            b_ptr += kBK;
            b_left -= kBK;
            return v;
        };
        // (the shifts do not change from step to step)
        constexpr bool kRows = MODE == GATHER_ROWS;  // (the other forms' units of A come in place)
        const uint32_t sh0 = kRows ? ((uint32_t)(uintptr_t)a_ptr0 & 3u) * 8u : 0u,
                       sh1 = kRows ? ((uint32_t)(uintptr_t)a_ptr1 & 3u) * 8u : 0u,
                       shb = ((uint32_t)(uintptr_t)b_ptr & 3u) * 8u;
        int left0 = a_left0, left1 = a_left1, leftb = b_left;

        // 64-byte swizzle: unit v of row r lies at unit v ^ ((r >> 1) & 3)
        const uint32_t a_at0 = (uint32_t)(row0 * kBK + ((u ^ ((row0 >> 1) & 3)) << 4));
        const uint32_t a_at1 = (uint32_t)(row1 * kBK + ((u1 ^ ((row1 >> 1) & 3)) << 4));
        const uint32_t b_at = (uint32_t)(b_row * kBK + ((b_u ^ ((b_row >> 1) & 3)) << 4));
        Units now = fetch();
        bool ok = true;
        int s = 0;
        uint32_t parity = 1;
        for (int step = 0; step < steps; ++step) {
            Units next = now;
            if (step + 1 < steps)
                next = fetch();
            ok = mbar_wait(&empty_bar[s], parity, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) {
                if (!*abort_flag) {
                    *abort_flag = 1;
                    atomicExch(p.status, ERR_PRODUCER_WAIT);
                }
                break;
            }
            *reinterpret_cast<uint4*>(tiles_a + s * kABytes + a_at0) = place(now.a0, sh0, kRows ? left0 : 16);
            *reinterpret_cast<uint4*>(tiles_a + s * kABytes + a_at1) = place(now.a1, sh1, kRows ? left1 : 16);
            *reinterpret_cast<uint4*>(tiles_b + s * kBBytes + b_at) = place(now.b, shb, leftb);
            left0 -= kBK, left1 -= kBK, leftb -= kBK;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                mbar_arrive(&full_bar[s]);
            now = next;
            if (++s == kStages) {
                s = 0;
                parity ^= 1u;
            }
        }
        if (ok) {
            ok = mbar_wait(&acc_full, 0, abort_flag);
            if (!ok && !*abort_flag) {
                *abort_flag = 1;
                atomicExch(p.status, ERR_EPILOGUE_WAIT);
            }
            ok = __all_sync(0xffffffffu, ok);
        }
        // (the loaders' barrier: `side` was written by one of them before the others' first step)
        asm volatile("bar.sync 1, %0;" ::"n"(kLoaders) : "memory");
        if (ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int q = warp & 3, half = warp >> 2;
            const int r = q * 32 + lane, mo = m0 + r;
            const int oimg = mo / pixels, opix = mo - oimg * pixels;
            // Channels that are no multiple of 4: a pixel's bytes go through shared memory (in place of the
            // operands, all of which have been read), so that a warp stores runs of adjacent bytes. A
            // byte per lane of 32 different pixels took 4 us a tile.
            constexpr int kPitch = 36;
            uint8_t* turn = smem + (size_t)warp * 32 * kPitch;
            const bool turned = MODE != GATHER_NCHW && (p.oc & 3) != 0 && !p.ep.acc_out && !p.ep.nchw_plane;
#pragma unroll 1
            for (int c = 0; c < 2; ++c) {
                const int col = half * 32 + c * 16;
                uint32_t v[16];
                __syncwarp();
                tmem_ld16(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)col, v);
                if (mo < p.m_total) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int c0 = n0 + col + 4 * j;
                        if (c0 >= p.oc)
                            break;
                        const int acc[4] = {(int)v[4 * j], (int)v[4 * j + 1], (int)v[4 * j + 2],
                                            (int)v[4 * j + 3]};
                        const QuadParams qp = side[(col >> 2) + j];
                        if constexpr (MODE == GATHER_NCHW) {
                            const uint32_t word = quad_values(acc, p.ep, qp, 0);
                            int8_t* out = p.dst + ((size_t)oimg * p.oc + c0) * pixels + opix;
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (c0 + i < p.oc)
                                    out[(size_t)i * pixels] = (int8_t)(word >> (8 * i));
                        } else {
                            const size_t off = (size_t)mo * p.oc + c0;
                            if (turned)
                                *reinterpret_cast<uint32_t*>(turn + lane * kPitch + c * 16 + 4 * j) =
                                        quad_values(acc, p.ep, qp, quad_z(p.ep, off, c0));
                            else if (p.ep.nchw_plane)
                                nchw_quad(acc, p.ep, qp, p.dst, off, c0);
                            else
                                epilogue_quad(acc, p.ep, qp, quad_z(p.ep, off, c0), p.dst, off, c0);
                        }
                    }
                }
            }
            if (turned) {
                __syncwarp();
                const int c0 = n0 + half * 32 + lane;
                int8_t* out = p.dst + (size_t)(m0 + q * 32) * p.oc + c0;
                const int rows = min(32, p.m_total - (m0 + q * 32));
                if (c0 < p.oc)
                    for (int i = 0; i < rows; ++i)
                        out[(size_t)i * p.oc] = (int8_t)turn[i * kPitch + lane];
            }
        }
    } else {
        // ---------------- MMA issuer (the whole warp waits, one lane issues) ----------------
        const uint32_t leader = elect_one() ? 1u : 0u;
        constexpr uint32_t idesc = umma_idesc_s8(kBM, kBN);
        const uint64_t da = umma_smem_desc(smem_u32(tiles_a), 16, 512, 4);
        const uint64_t db = umma_smem_desc(smem_u32(tiles_b), 16, 512, 4);
        const uint32_t a_hi = (uint32_t)(da >> 32), b_hi = (uint32_t)(db >> 32);
        uint32_t a_lo = (uint32_t)da, b_lo = (uint32_t)db, phase = 0;
        int s = 0;
        bool ok = true;
        for (int step = 0; step < steps; ++step) {
            ok = mbar_wait(&full_bar[s], phase, abort_flag);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok)
                break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            umma_s8(leader, tmem_base, a_lo, a_hi, b_lo, b_hi, idesc, step != 0);
            if (step * kBK + 32 < p.k_total)
                umma_s8(leader, tmem_base, a_lo + 2, a_hi, b_lo + 2, b_hi, idesc, 1);
            umma_commit_if(leader, smem_u32(&empty_bar[s]));
            a_lo += kABytes / 16;
            b_lo += kBBytes / 16;
            if (++s == kStages) {
                s = 0;
                phase ^= 1u;
                a_lo = (uint32_t)da;
                b_lo = (uint32_t)db;
            }
        }
        if (ok) {
            umma_commit_if(leader, smem_u32(&acc_full));
        } else if (!*abort_flag) {
            *abort_flag = 1;
            atomicExch(p.status, ERR_MMA_WAIT);
        }
        __syncwarp();
    }

    // ---------------- teardown ----------------
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag) {
        // a wait ran out: let MMAs retire (bounded) before shared memory and TMEM are given back
        if (warp == kLoaders / 32 && lane == 0) {
            umma_commit(&drain_bar);
            const long long t0 = clock64();
            while (!mbar_try_wait(&drain_bar, 0)) {
                if (clock64() - t0 > kWaitCycles) {
                    atomicExch(p.status, ERR_DRAIN_WAIT);
                    break;
                }
            }
        }
        __syncthreads();
    }
    if (warp == kLoaders / 32) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kBN)
                     : "memory");
    }
}

template <int MODE>
int launch_mode(const GatherParams& p, int grid, cudaStream_t st) {
    static KernelReady ready;
    if (!ready.smem(conv_gather_kernel<MODE>, kSmem))
        return check_launch("conv_gather smem attribute");
    if (tuning().debug)
        fprintf(stderr, "conv_gather<%d>: grid %d k %d\n", MODE, grid, p.k_total);
    const size_t outputs = (size_t)p.m_total * p.oc;
    const Writes writes = p.ep.acc_out ? Writes{p.ep.acc_out, outputs * 4} : Writes{p.dst, outputs};
    launch_pdl(writes, conv_gather_kernel<MODE>, dim3(grid), dim3(kThreads), (size_t)kSmem, st, p);
    return check_launch("conv_gather");
}

// the form that fetches this source, -1: none
int gather_mode(const ConvArgs& a, const int8_t* src, bool nchw) {
    if (nchw)
        return a.kh * a.kw <= kMaxTaps ? GATHER_NCHW : -1;
    if (a.kh == 1 && a.kw == 1 && a.sh == 1 && a.sw == 1 && a.ph == 0 && a.pw == 0)
        return GATHER_ROWS;
    if (a.ic % 16 == 0 && ((uintptr_t)src & 15) == 0)
        return GATHER_VEC16;
    return a.ic % 4 == 0 && ((uintptr_t)src & 3) == 0 ? GATHER_WORDS : -1;
}

}  // namespace

// nchw: the reference's layouts (NCHW source and result, OIHW filter); else NHWC with the packed filter.
// Everything the kernel computes with is checked here; operands of any alignment are taken.
bool conv_gather_supported(const ConvArgs& a, const int8_t* src, bool nchw) {
    if (a.groups != 1 || a.src_is_nchw || a.true_division || (nchw && a.z))
        return false;
    const long long k = (long long)a.ic * a.kh * a.kw;
    const long long tiles = ((long long)a.m + kBM - 1) / kBM * ((a.oc + kBN - 1) / kBN);
    if (k >= 1 << 30 || tiles >= 1ll << 31)
        return false;
    return gather_mode(a, src, nchw) >= 0;
}

// Against one CUDA thread per output value (NHWC): a tile's start and end are 3 us, so products of
// less than 2^20 terms stay there (336 x 32 over K = 36 7.9 us there, 9.0 here; 1332 x 196 over 847 329 and
// 16). Against re-laying both tensors (NCHW): a step of byte loads takes 3 us, so at most two, and not
// where the GPU is full with them (11970 x 40 over 24 20.2 and 9.6, 9537 x 16 over 128 15.4 and 12.4;
// 16616 x 128 over 64, 260 tiles, 12.7 and 15.0).
bool conv_gather_pays(const ConvArgs& a, bool nchw) {
    if (tuning().gather != 1)
        return tuning().gather == 2;
    const long long k = (long long)a.ic * a.kh * a.kw;
    const long long tiles = ((long long)a.m + kBM - 1) / kBM * ((a.oc + kBN - 1) / kBN);
    if (nchw)
        return (k <= kBK && tiles <= sm_count()) || (k <= 2 * kBK && a.oc <= kBN && 2 * tiles <= sm_count());
    return (long long)a.m * a.oc * k >= 1ll << 20;
}

int launch_conv_gather(
        const ConvArgs& a, bool nchw, const int8_t* src, const int8_t* flt, const int32_t* bias,
        const float* flt_scales, int8_t* dst, cudaStream_t st) {
    GatherParams p;
    p.src = src;
    p.flt = flt;
    p.m_total = a.m;
    p.oc = a.oc;
    p.k_total = a.ic * a.kh * a.kw;
    p.src_bytes = (size_t)a.n * a.ih * a.iw * a.ic;
    p.flt_bytes = (size_t)a.oc * p.k_total;
    p.ic = a.ic;
    p.ih = a.ih;
    p.iw = a.iw;
    p.oh = a.oh;
    p.ow = a.ow;
    p.kh = a.kh;
    p.kw = a.kw;
    p.sh = a.sh;
    p.sw = a.sw;
    p.ph = a.ph;
    p.pw = a.pw;
    p.dh = a.dh;
    p.dw = a.dw;
    p.n_tiles = (a.oc + kBN - 1) / kBN;
    p.src_vec = a.ic % 16 == 0 && ((uintptr_t)src & 15) == 0;
    p.flt_vec = p.k_total % 16 == 0 && ((uintptr_t)flt & 15) == 0;
    fill_epilogue(a, bias, flt_scales, &p.ep);
    p.dst = dst;
    p.status = device_status_word(st);
    if (!p.status)
        return ST_MALLOC;
    const int grid = ((a.m - 1) / kBM + 1) * p.n_tiles;  // (a.m may be as large as an int holds)
    switch (gather_mode(a, src, nchw)) {
        case GATHER_VEC16: return launch_mode<GATHER_VEC16>(p, grid, st);
        case GATHER_WORDS: return launch_mode<GATHER_WORDS>(p, grid, st);
        case GATHER_ROWS: return launch_mode<GATHER_ROWS>(p, grid, st);
        case GATHER_NCHW: return launch_mode<GATHER_NCHW>(p, grid, st);
    }
    return set_error(ST_NO_IMPLEMENT, "ConvBias with gathered operands does not apply to this shape");
}

}  // namespace mb200
