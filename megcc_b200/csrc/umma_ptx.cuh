// Inline-PTX building blocks shared by the tensor-core ConvBias kernels: mbarrier waits with
// a time limit, TMA loads (tiled and im2col; no cluster multicast is used anywhere), UMMA
// shared-memory / instruction descriptors, tcgen05.mma / commit / ld.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <mutex>

#ifndef MB200_TRY_WAIT_HINT_NS
#define MB200_TRY_WAIT_HINT_NS 2000
#endif
#ifndef MB200_WAIT_SLEEP_CAP
#define MB200_WAIT_SLEEP_CAP 160
#endif
namespace mb200 {
namespace umma {

constexpr long long kWaitCycles = 1LL << 31;  // ~1 s: only a lost barrier gets there

enum : int {
    ERR_PRODUCER_WAIT = 0x101,
    ERR_MMA_WAIT = 0x102,
    ERR_EPILOGUE_WAIT = 0x103,
    ERR_DRAIN_WAIT = 0x104,
    ERR_MMA_ACC_WAIT = 0x105,
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

// The warp index as a value the compiler knows to be the same in all lanes, and one lane chosen
// by the hardware. A role that runs as a whole warp and only issues under `if (leader)` keeps
// its descriptors and addresses in uniform registers, where tcgen05.mma takes them from; in a
// `lane == 0` branch every operand is moved there first, instruction by instruction (measured
// alone, tf32 with A in tensor memory: 128 x 32 x 8 in 16 clocks against 45, 128 x 64 in 32
// against 45).
__device__ __forceinline__ int uniform_warp_index() {
    return __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
}
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "elect.sync _|p, 0xffffffff;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(r));
    return r != 0;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
            "{\n\t.reg .pred p;\n\t"
            // the hint lets the hardware park the thread until the phase completes (or the
            // time passes) instead of burning issue slots in a software spin
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity), "r"((uint32_t)MB200_TRY_WAIT_HINT_NS)
            : "memory");
    return ok != 0;
}

// Bounded wait. Returns false when the limit ran out or another role already gave up.
__device__ __forceinline__ bool mbar_wait(
        uint64_t* bar, uint32_t parity, volatile int* abort_flag,
        long long limit = kWaitCycles) {
    // A few immediate polls, then short sleeps (20 ns doubling to 160 ns): roles that wait
    // for most of a kernel (producer and MMA thread of an epilogue-bound layer) should not
    // take issue slots from the warps that work. Measured against polling without sleeps on
    // one GPU, neither way changed any kernel's time by more than 1 %.
#pragma unroll 1
    for (int i = 0; i < 8; ++i)
        if (mbar_try_wait(bar, parity))
            return true;
    const long long t0 = clock64();
    unsigned ns = 20;
    for (int spin = 0;; ++spin) {
        if (mbar_try_wait(bar, parity))
            return true;
        __nanosleep(ns);
        if (ns < MB200_WAIT_SLEEP_CAP)
            ns *= 2;
        if ((spin & 63) == 63) {
            if (*abort_flag)
                return false;
            if (clock64() - t0 > limit)
                return false;
        }
    }
}

// The same on a shared-memory address: no generic pointer is converted per call.
__device__ __forceinline__ bool mbar_try_wait_u32(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity), "r"((uint32_t)MB200_TRY_WAIT_HINT_NS)
            : "memory");
    return ok != 0;
}

// One try in line (a loop that is seldom late spends its instructions there), the bounded wait
// behind it out of line.
static __device__ __noinline__ bool mbar_wait_slow(
        uint32_t bar, uint32_t parity, volatile int* abort_flag, long long limit) {
    const long long t0 = clock64();
    unsigned ns = 20;
#pragma unroll 1
    for (int spin = 0;; ++spin) {
        if (mbar_try_wait_u32(bar, parity))
            return true;
        if (spin >= 8) {
            __nanosleep(ns);
            if (ns < MB200_WAIT_SLEEP_CAP)
                ns *= 2;
        }
        if ((spin & 63) == 63) {
            if (*abort_flag)
                return false;
            if (clock64() - t0 > limit)
                return false;
        }
    }
}
__device__ __forceinline__ bool mbar_wait_u32(
        uint32_t bar, uint32_t parity, volatile int* abort_flag, long long limit = kWaitCycles) {
    return mbar_try_wait_u32(bar, parity) || mbar_wait_slow(bar, parity, abort_flag, limit);
}

// brings a tensor map (a kernel parameter) into the descriptor cache ahead of its first use
__device__ __forceinline__ void tma_prefetch_map(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"((uint64_t)map) : "memory");
}

// ---- thread-block clusters ----
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// The two halves of a barrier for every thread of every CTA of the cluster, for work in between
// that needs nobody
__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Asks for the line of `p` ahead of its use: the value is thrown away, its line stays in the L1.
// keep() takes it (the load is not dropped, and is not waited for before that).
__device__ __forceinline__ uint32_t ask_for(const void* p) {
    uint32_t v;
    asm volatile("ld.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void keep(uint32_t v) {
    asm volatile("" ::"r"(v) : "memory");
}
// 16 bytes at the shared-memory address `local` of CTA `rank`
__device__ __forceinline__ uint4 ld_cluster_v4(uint32_t local, int rank) {
    uint32_t addr;
    uint4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(local), "r"(rank));
    asm volatile("ld.shared::cluster.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(addr)
                 : "memory");
    return v;
}

__device__ __forceinline__ void tma_load_2d(
        void* smem, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
    asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(smem)),
            "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
            : "memory");
}

__device__ __forceinline__ void tma_load_3d(
        void* smem, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(smem)),
            "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
            : "memory");
}

__device__ __forceinline__ void tma_load_4d(
        void* smem, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3) {
    asm volatile(
            "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(smem)),
            "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
            : "memory");
}

__device__ __forceinline__ void tma_load_5d(
        void* smem, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2, int c3, int c4) {
    asm volatile(
            "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(smem_u32(smem)),
            "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
            : "memory");
}

__device__ __forceinline__ void tma_load_im2col_4d(
        void* smem, const CUtensorMap* map, uint64_t* bar, int c, int w, int h, int n,
        uint16_t off_w, uint16_t off_h) {
    asm volatile(
            "cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};" ::"r"(smem_u32(smem)),
            "l"((uint64_t)map), "r"(smem_u32(bar)), "r"(c), "r"(w), "r"(h), "r"(n), "h"(off_w),
            "h"(off_h)
            : "memory");
}

// The same from a converged warp: carried out by the lane whose `leader` is non-zero. A role that
// runs as a whole warp keeps its addresses and coordinates in uniform registers, where the
// instruction wants them; inside a one-lane branch each is moved there first.
__device__ __forceinline__ void mbar_expect_tx_if(uint32_t leader, uint32_t bar, uint32_t bytes) {
    asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
            "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar),
            "r"(bytes), "r"(leader)
            : "memory");
}
__device__ __forceinline__ void tma_load_2d_if(
        uint32_t leader, uint32_t smem, const CUtensorMap* map, uint32_t bar, int c0, int c1) {
    asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
            "@q cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4}], [%2];\n\t}" ::"r"(smem),
            "l"((uint64_t)map), "r"(bar), "r"(c0), "r"(c1), "r"(leader)
            : "memory");
}
__device__ __forceinline__ void tma_load_im2col_4d_if(
        uint32_t leader, uint32_t smem, const CUtensorMap* map, uint32_t bar, int c, int w, int h,
        int n, uint16_t off_w, uint16_t off_h) {
    asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %9, 0;\n\t"
            "@q cp.async.bulk.tensor.4d.shared::cluster.global.im2col.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%3, %4, %5, %6}], [%2], {%7, %8};\n\t}" ::"r"(smem),
            "l"((uint64_t)map), "r"(bar), "r"(c), "r"(w), "r"(h), "r"(n), "h"(off_w), "h"(off_h),
            "r"(leader)
            : "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile.
//   swizzled (64 B): rows of 64 bytes, 8-row groups `sbo` bytes apart, `lbo` unused
//   plain:           8x16-byte core matrices; `lbo` = distance between the two 16-byte K
//                    halves of one MMA, `sbo` = distance between 8-row groups
__device__ __forceinline__ uint64_t umma_smem_desc(
        uint32_t saddr, uint32_t lbo, uint32_t sbo, uint32_t layout_type) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version of sm_100
    d |= (uint64_t)layout_type << 61;
    return d;
}

// kind::i8 instruction descriptor: int32 accumulate, signed 8-bit A and B, both K-major.
__host__ __device__ constexpr uint32_t umma_idesc_s8(int m, int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}

// Issued by the lane whose `leader` is non-zero, without a branch. Descriptors come as their low
// words (address field and leading-dimension offset, the part that moves from step to step)
// and constant high words.
__device__ __forceinline__ void umma_s8(
        uint32_t leader, uint32_t tmem_d, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
        uint32_t idesc, uint32_t accumulate) {
    asm volatile(
            "{\n\t.reg .pred p, q;\n\t.reg .b64 a, b;\n\t"
            "mov.b64 a, {%1, %2};\n\tmov.b64 b, {%3, %4};\n\t"
            "setp.ne.b32 p, %6, 0;\n\tsetp.ne.b32 q, %7, 0;\n\t"
            "@q tcgen05.mma.cta_group::1.kind::i8 [%0], a, b, %5, p;\n\t}" ::"r"(tmem_d),
            "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(accumulate), "r"(leader)
            : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile(
            "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                    smem_u32(bar))
            : "memory");
}

// tcgen05.commit by the lane whose `leader` is non-zero (no branch around it)
__device__ __forceinline__ void umma_commit_if(uint32_t leader, uint32_t bar) {
    asm volatile(
            "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
            "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(
                    bar),
            "r"(leader)
            : "memory");
}

// Loads of tensor memory are the whole warp's (.aligned). Where its lanes part between two of them (pixels
// beyond the result store nothing), nothing but a __syncwarp() in front of the second brings them together.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
            "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
            "[%32];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
              "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
              "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
              "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]),
              "=r"(v[31])
            : "r"(taddr)
            : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}


// 16 columns, load and wait in one statement
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
            "tcgen05.wait::ld.sync.aligned;"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
              "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(taddr)
            : "memory");
}

// 16 columns, WITHOUT waiting: the registers may be read only after tmem_ld_wait16(v)
__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
            : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
              "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
              "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
            : "r"(taddr)
            : "memory");
}

// Waits for this thread's TMEM loads. The registers are named as in/out operands so that
// the compiler cannot move a use of them above the wait.
__device__ __forceinline__ void tmem_ld_wait16(uint32_t (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]),
                   "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]), "+r"(v[10]), "+r"(v[11]),
                   "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15])
                 :
                 : "memory");
}

__device__ __forceinline__ uint32_t pack4_prmt(int a, int b, int c, int d) {
    const uint32_t ab = __byte_perm((uint32_t)a, (uint32_t)b, 0x0040);
    const uint32_t cd = __byte_perm((uint32_t)c, (uint32_t)d, 0x0040);
    return __byte_perm(ab, cd, 0x5410);
}

// driver entry points for tensor-map encoding, resolved once at run time
typedef CUresult (*EncodeTiledFn)(
        CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
        const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
        CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*EncodeIm2colFn)(
        CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
        const cuuint64_t*, const int*, const int*, cuuint32_t, cuuint32_t, const cuuint32_t*,
        CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
        CUtensorMapFloatOOBfill);

struct DriverApi {
    EncodeTiledFn tiled = nullptr;
    EncodeIm2colFn im2col = nullptr;
    bool ok = false;
};

inline const DriverApi& driver_api() {
    static DriverApi api = [] {
        DriverApi a;
        cudaDriverEntryPointQueryResult q;
        void* f = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) ==
                    cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            a.tiled = (EncodeTiledFn)f;
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &f, cudaEnableDefault, &q) ==
                    cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            a.im2col = (EncodeIm2colFn)f;
        a.ok = a.tiled && a.im2col;
        return a;
    }();
    return api;
}

inline int sm_count() {
    static int sms[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64)
        return 148;
    if (!sms[dev]) {
        int v = 0;
        if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0)
            v = 148;
        sms[dev] = v;
    }
    return sms[dev];
}

// Remembers, per device, that a kernel was allowed `bytes` of dynamic shared memory: the
// attribute call costs a launch about a microsecond. One static object per kernel instantiation.
// A kernel may ask for different sizes, from several threads: the attribute only ever grows,
// and what is remembered is never more than what is set.
struct KernelReady {
    std::atomic<int> bytes_set[64] = {};
    std::mutex mu;
    template <class Kernel>
    bool smem(Kernel kernel, int bytes) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess)
            return false;
        if (dev >= 0 && dev < 64 && bytes_set[dev].load(std::memory_order_relaxed) >= bytes)
            return true;
        std::lock_guard<std::mutex> lock(mu);
        if (dev >= 0 && dev < 64 && bytes_set[dev].load(std::memory_order_relaxed) >= bytes)
            return true;
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) !=
            cudaSuccess)
            return false;
        if (dev >= 0 && dev < 64)
            bytes_set[dev].store(bytes, std::memory_order_relaxed);
        return true;
    }
};

// Clusters of `size` CTAs (one per SM) that the GPU holds at once: whole clusters live inside a
// GPC, so for eight it is less than sm_count() / 8. Asked once per kernel, size and device.
struct ClusterCapacity {
    std::atomic<int> known[64][4] = {};
    template <class Kernel>
    int clusters(Kernel kernel, int size, int threads, int dynamic_smem) {
        const int k = size == 2 ? 1 : size == 4 ? 2 : size == 8 ? 3 : 0;
        int dev = 0;
        if (k == 0 || cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
            return 0;
        int n = known[dev][k].load(std::memory_order_relaxed);
        if (n == 0) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3((unsigned)(sm_count() / size * size));
            cfg.blockDim = dim3((unsigned)threads);
            cfg.dynamicSmemBytes = (size_t)dynamic_smem;
            cudaLaunchAttribute attr;
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = (unsigned)size;
            attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess || n <= 0) {
                cudaGetLastError();
                n = sm_count() / size * 3 / 4;
            }
            known[dev][k].store(n, std::memory_order_relaxed);
        }
        return n;
    }
};

// CTAs of `threads` threads that one SM holds at once, from the kernel's register count,
// its dynamic shared memory and its TMEM columns. (The runtime's occupancy query answers 1
// for these kernels whatever their footprint, so the arithmetic is done here.)
template <class Kernel>
inline int resident_ctas_per_sm(Kernel kernel, int threads, int dynamic_smem, int tmem_cols) {
    cudaFuncAttributes fa;
    int regs = 128;
    if (cudaFuncGetAttributes(&fa, kernel) == cudaSuccess && fa.numRegs > 0)
        regs = fa.numRegs;
    const int regs_per_warp = (regs * 32 + 511) / 512 * 512;  // allocation granularity
    const int warps = (threads + 31) / 32;
    int by_regs = 65536 / (regs_per_warp * warps);
    int by_smem = (227 * 1024) / (dynamic_smem + 1024);
    int by_tmem = tmem_cols > 0 ? 512 / tmem_cols : 32;
    int n = by_regs < by_smem ? by_regs : by_smem;
    n = n < by_tmem ? n : by_tmem;
    return n < 1 ? 1 : n;
}

// resident_ctas_per_sm, asked once per kernel, shared-memory size and device (a function-attribute
// query on every launch costs it about a microsecond)
struct ResidentCtas {
    std::atomic<long long> known[64] = {};  // shared memory << 8 | CTAs
    template <class Kernel>
    int per_sm(Kernel kernel, int threads, int dynamic_smem, int tmem_cols) {
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
            return resident_ctas_per_sm(kernel, threads, dynamic_smem, tmem_cols);
        const long long k = known[dev].load(std::memory_order_relaxed);
        if (k && (k >> 8) == dynamic_smem)
            return (int)(k & 255);
        const int n = resident_ctas_per_sm(kernel, threads, dynamic_smem, tmem_cols);
        known[dev].store(((long long)dynamic_smem << 8) | n, std::memory_order_relaxed);
        return n;
    }
};

}  // namespace umma
}  // namespace mb200
