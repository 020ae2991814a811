// qint8 ConvBias as implicit GEMM on the sm_100a tensor cores.
//
//   D[m, oc] = sum_{fy,fx,c} A[m, (fy,fx,c)] * W[oc, (fy,fx,c)],   m = (n, oh, ow) linearised
//
// * activations NHWC int8. One TMA im2col load brings, for one filter tap, the channels of
//   the 128 consecutive output pixels of a tile straight into a K-major shared-memory tile;
//   padding and stride are resolved by the im2col bounding box and traversal stride.
// * filter pre-packed K-major [OC][taps][channels], fetched by tiled 2D TMA.
// * tcgen05.mma kind::i8, M=128 x N=BN x K=32 per instruction, int32 accumulators in TMEM,
//   two accumulator buffers so the epilogue of one tile overlaps the MMAs of the next.
// * persistent CTAs walk the tile list; warp 0 = TMA producer, warp 1 = MMA issuer (+ TMEM
//   alloc), warps 2..9 = epilogue (tcgen05.ld -> +bias -> fp32 requantisation in the
//   reference's operation order -> activation -> int8 -> 16-byte stores).
// * every wait is bounded: when it runs out the kernel records a code in the device status
//   word, drains what it started, frees its TMEM and returns.
//
// Two operand geometries:
//   WIDE  one tap x 64 or 128 channels per pipeline stage, 64- / 128-byte swizzle (input channels
//         % 16 == 0, at least 64 with a spatial filter or a stride)
//   TAP16 four taps x 16 channels per stage, no swizzle: the form a stride-2 convolution with
//         at most 4 input channels takes after a 2x2 space-to-depth step (see conv_s2d.cu)
//
// Replaces the loop nest of compiler/lib/KernelGen/BareMetal/ConvKernel.cpp:305-344 and
// its epilogue (:374-382, BareMetal/Activation.cpp:105-113).
#include <map>
#include <mutex>
#include <utility>

#include "conv_umma_kernel.cuh"

namespace mb200 {

using namespace umma;
using namespace umma_conv;

namespace umma_conv {
extern template int launch_kernel<64, GEOM_WIDE>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
extern template int launch_kernel<64, GEOM_WIDE128>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
extern template int launch_form<64, GEOM_TAP16>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
extern template int umma_clusters<64, GEOM_WIDE>(int);
extern template int umma_clusters<64, GEOM_WIDE128>(int);
extern template int launch_kernel<128, GEOM_WIDE>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
extern template int launch_kernel<128, GEOM_WIDE128>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
extern template int launch_form<128, GEOM_TAP16>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
extern template int launch_kernel<256, GEOM_WIDE128>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
extern template int launch_form<256, GEOM_WIDE128, true>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
}  // namespace umma_conv

namespace {

// A layer with fewer tiles than SMs (a small batch): 64- or 128-column tiles, and how many CTAs
// of a cluster share a tile's K loop. The pair with the shortest estimated chain of its
// busiest CTA, in clocks: a pipeline step of 128-byte rows (half of that for 64-byte ones) costs
// 300 with 64 columns and 380 with 128, a tile's end 1200 and 1800 (3000 more where the channels
// are no multiple of 32 and take the general epilogue); the exchange of the shares over the
// cluster 2200 and 350 for every four channels that a thread then finishes. A split has to
// promise a sixth less, and only 64-column tiles are split: with 128 every exchange is twice as
// long. Measured per call, 256 -> 256 3x3 with a residual step over five images of 14 x 14: 7.6 us as
// 32 tiles of 64 columns split in four, 9.1 unsplit, 11.0 as 16 tiles of 128 split in four;
// 512 -> 512 over one of 7 x 7: 5.8 split in eight, 13.9 unsplit; 128 -> 128 over two of 28 x 28: 6.1
// split in four, 5.3 unsplit; a 512 -> 1000 classifier: 3.7 split in two, 4.9 unsplit.
// Over 160 layers that are in no network here (1x1 and 3x3, strides 1 and 2, 64 to 1024 channels to 64
// to 1024, 25 to 10000 pixels): never more than 3 % slower than the unsplit tile that was taken before
// this estimate, 8 % on average behind the best of all widths and splits, at most 75 %. Those farthest
// off are 3x3 layers over 320 channels (64-byte rows are priced at half of 128-byte ones and cost
// more) and 1x1 layers with 20 to 50 row tiles, where 64 columns unsplit would be up to 34 % faster
// than the 128 taken.
void choose_split(int m_tiles, int oc, int k_iters, bool wide128, int sms, int* bn, int* csplit) {
    long long best = -1;
    const int bn_first = *bn;
    for (int b = 64; b <= 128; b *= 2) {
        if (b > 64 && oc <= 64)
            break;
        const long long tiles = (long long)m_tiles * ((oc + b - 1) / b);
        const int step = (b == 128 ? 380 : 300) / (wide128 ? 1 : 2);
        for (int s = 1; s <= 8; s *= 2) {
            if (s > 1) {
                if (b > 64)
                    break;
                const int fit = wide128 ? umma_clusters<64, GEOM_WIDE128>(s)
                                        : umma_clusters<64, GEOM_WIDE>(s);
                if (k_iters / s < 2 || tiles > fit || tiles * s > sms)
                    break;
            }
            const long long waves = (tiles * s + sms - 1) / sms;
            const long long steps = (long long)((k_iters + s - 1) / s) * step;
            const int quads = b / (8 * s) > 1 ? b / (8 * s) : 1;
            const int end = (b == 128 ? 1800 : 1200) + (oc % 32 ? 3000 : 0);
            const long long clocks = s > 1 ? (steps + 2200 + 350 * quads) * 6 / 5
                                           : waves * (steps + end);
            // (a tie goes to the width the caller had chosen)
            if (best < 0 || clocks < best || (clocks == best && b == bn_first && s == 1)) {
                best = clocks;
                *bn = b;
                *csplit = s;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// split-K for the last, partly filled wave of 128 x 256 tiles
// ------------------------------------------------------------------------------------------
// 196 tiles on 148 SMs take two waves with the second a third full. The tiles of that last
// wave can be cut along K into `split` parts, each a work item of its own, so that the wave
// takes 1/split of a tile's MMA time when the parts fit the SMs. Parts leave their int32
// accumulators in scratch slabs; the last part of a tile to finish sums them and runs the
// usual epilogue (integer sums: the result does not depend on the order).
//
// OFF unless MB200_CONV_SPLITK=2..4 asks for it: bit-exact, but measured SLOWER on the
// ResNet-18 layers at batch 256 (512->512 7x7: 30.5 -> 32.6 us; 256->256 14x14: 26.7 ->
// 41.4 us). A part of 6-12 pipeline steps is 2-5 us of MMAs, while its epilogue writes a
// 128 KB slab (four times the int8 tile) and the finisher reads `split` slabs back from L2
// with eight 16-byte loads in flight per thread: about 64 KB in flight per SM, some 6 us for
// 384 KB, all of it after the last MMA of the kernel with nothing left to overlap it.
constexpr int kMaxSplitItems = 2 * 148;
constexpr size_t kSlabBytes = (size_t)kBM * 256 * 4;
constexpr size_t kCounterBytes = 4096;  // one word per split tile (fewer than 148)
constexpr size_t kSplitScratchBytes = kCounterBytes + kMaxSplitItems * kSlabBytes;

struct SplitPlan {
    int full_tiles, split, k_per_part, total_items;
};

SplitPlan plan_split_k(int tiles, int k_iters, int ctas) {
    SplitPlan sp{tiles, 1, k_iters, tiles};
    const int forced = tuning().conv_splitk;  // 2..4: that split wherever it fits
    if (forced < 2 || ctas <= 0)
        return sp;
    const int rem = tiles % ctas;
    if (rem == 0)
        return sp;
    int best = 1;
    for (int s = 2; s <= 4; ++s) {
        const int per_part = (k_iters + s - 1) / s;
        if (k_iters / s < 4 || (s - 1) * per_part >= k_iters ||  // no short or empty part
            rem * s > kMaxSplitItems || rem > (int)(kCounterBytes / 4))
            continue;
        if (forced == s)
            best = s;
    }
    if (best > 1) {
        sp.full_tiles = tiles - rem;
        sp.split = best;
        sp.k_per_part = (k_iters + best - 1) / best;
        sp.total_items = sp.full_tiles + rem * best;
    }
    return sp;
}

// Scratch for the slabs: one buffer per (device, stream), so that launches on different
// streams cannot meet in it; allocated at first use, never while the stream is capturing
// (the caller then runs unsplit). The counters at its start are zeroed once: every launch
// leaves them at zero.
void* split_scratch(cudaStream_t st) {
    static std::mutex mu;
    static std::map<std::pair<int, cudaStream_t>, void*> pool;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess)
        return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    auto it = pool.find(std::make_pair(dev, st));
    if (it != pool.end())
        return it->second;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return nullptr;
    }
    void* ptr = nullptr;
    if (cudaMalloc(&ptr, kSplitScratchBytes) != cudaSuccess ||
        cudaMemset(ptr, 0, kCounterBytes) != cudaSuccess) {
        cudaGetLastError();
        if (ptr)
            cudaFree(ptr);
        ptr = nullptr;
    }
    pool[std::make_pair(dev, st)] = ptr;
    return ptr;
}

}  // namespace

// 1x1 filter, stride 1, no padding, NHWC: the convolution is a matrix product over the
// activation as it lies in memory
static bool conv_is_plain_matrix(const ConvArgs& a) {
    return a.kh == 1 && a.kw == 1 && a.sh == 1 && a.sw == 1 && a.ph == 0 && a.pw == 0 &&
           !a.src_is_nchw;
}

bool conv_umma_supported(
        const ConvArgs& a, const int8_t* src, const int8_t* flt, const int8_t* dst) {
    if (a.groups != 1 || a.src_is_nchw)
        return false;
    // rows start on 16-byte boundaries; an im2col map asks for boxes no wider than the tensor
    if (a.ic % 16 != 0 || (a.ic < kBK && !conv_is_plain_matrix(a)))
        return false;
    if (a.kh * a.kw > 49 || a.dh != 1 || a.dw != 1)
        return false;
    // im2col bounding-box corners and tap offsets are 8-bit fields for a 4-D map
    if (a.ph > 64 || a.pw > 64 || a.kh > 64 || a.kw > 64 || a.sh > 8 || a.sw > 8)
        return false;
    // im2col maps are built over at least 128 KiB (descriptor_images); a pointwise
    // convolution uses a tiled map over the plain matrix and has no such limit
    if (!conv_is_plain_matrix(a) && descriptor_images(a, src) == 0)
        return false;
    if (((uintptr_t)src | (uintptr_t)flt | (uintptr_t)dst) & 15)
        return false;
    return true;
}

// geom: 0 = WIDE (src NHWC with ic % 16 == 0, filter [OC][KH][KW][IC]). Where the channels are no whole
//           number of a stage's rows, the load fills the rest of the last row with zeros: a
//           704 x 5920 x 7328 product takes 27 us that way, 12577 on one CUDA thread per output;
//       1 = TAP16 (src NHWC with exactly 16 channels, stride 1, filter [OC][taps][16] with the
//           tap count a multiple of 4; `a` then describes that transformed convolution, with
//           a.ph/a.pw the LOW padding and a.oh/a.ow the output extent)
int launch_conv_umma_geom(
        const ConvArgs& a, int geom_in, const int8_t* src, const int8_t* flt, const int32_t* bias,
        const float* flt_scales, int8_t* dst, cudaStream_t st) {
    int geom = geom_in;
    const DriverApi& api = driver_api();
    if (!api.ok)
        return set_error(ST_RUNTIME, "cuTensorMapEncode* entry points not found in the driver");
    const int taps = a.kh * a.kw;
    if (geom == GEOM_TAP16 && (a.ic != 16 || taps % 4 != 0 || a.sh != 1 || a.sw != 1))
        return set_error(ST_INVALID_LAYOUT, "TAP16 geometry needs 16 channels and 4k taps");
    if (((uintptr_t)bias & 15) || ((uintptr_t)flt_scales & 15))
        return set_error(ST_INVALID_LAYOUT, "bias and channel scales must be 16-byte aligned");

    // 128-channel rows (fewer, larger TMA requests) wherever they do not hold more padding than
    // 64-channel ones, and from 512 channels on, where another half row of zeros is at most an eighth
    // of the K loop
    const int half_rows = (a.ic + kBK - 1) / kBK;
    if (geom == GEOM_WIDE && (half_rows % 2 == 0 || a.ic >= 512) &&
        (a.ic >= 128 || conv_is_plain_matrix(a)) && tuning().wide128)
        geom = GEOM_WIDE128;
    // MB200_CONV_PAIR=1: one 256 x 256 tile per pair of SMs (conv_pair.cu) wherever it applies.
    // Off by default: both kernels are bound by shared-memory bandwidth (operand reads of
    // the MMAs plus the TMA writes), and on the ResNet layers the pair measured no faster
    // than the 128 x 256 tile of a single SM.
    if (geom == GEOM_WIDE128 && conv_pair_supported(a, src, flt, dst)) {
        if (tuning().conv_pair != 0)
            return launch_conv_pair(a, src, flt, bias, flt_scales, dst, st);
    }
    const int chans = geom == GEOM_WIDE128 ? 128 : geom == GEOM_WIDE ? kBK : 16;
    int bn = a.oc <= 64 ? 64 : 128, csplit = 1;
    {
        // 256 output channels per tile when the K loop is long enough to hide the epilogue
        // of a single CTA per SM and the busiest SM is done earlier: a step of 128 bytes takes 745
        // clocks with 256 columns and 512 with 128 (operand reads and TMA writes share the SM's
        // shared-memory port). Measured: 4096 x 1000 x 2048 (128 tiles of 256 columns, 256 of 128) 12.3
        // against 13.3 us, 704 x 5920 x 7328 (144, 282) 29.7 against 34.2; 1696 x 1088 x 3040 (70, 126)
        // 14.9 against 12.0.
        const long long k_bytes = (long long)taps * a.ic;
        const long long m_tiles = (a.m - 1) / kBM + 1;
        const long long sms = sm_count();
        const long long busiest256 = (m_tiles * ((a.oc + 255) / 256) + sms - 1) / sms;
        const long long busiest128 = (m_tiles * ((a.oc + 127) / 128) + sms - 1) / sms;
        const int force = tuning().conv_bn;
        if (geom == GEOM_WIDE128 && a.oc > 128 && k_bytes >= 1024 &&
            busiest256 * 745 < busiest128 * 512)
            bn = 256;
        if (force == 256 && geom == GEOM_WIDE128 && a.oc > 128)
            bn = 256;
        if (force == 128 && a.oc > 64)
            bn = 128;
        // A short K loop leaves the kernel to its epilogue warps: 64-column tiles hold half
        // the TMEM, so three CTAs (24 epilogue warps) fit an SM instead of two
        if (force == 64 || (force == 0 && k_bytes <= 256 && bn == 128))
            bn = 64;
        // fewer tiles than SMs: narrower tiles, K split over clusters
        const long long tiles = (long long)((a.m - 1) / kBM + 1) * ((a.oc + bn - 1) / bn);
        const int k_iters = geom == GEOM_TAP16 ? taps / 4 : taps * ((a.ic + chans - 1) / chans);
        if (geom != GEOM_TAP16 && bn <= 128 && force == 0 && a.test_wait_cycles == 0 &&
            tiles <= sms)
            choose_split((a.m - 1) / kBM + 1, a.oc, k_iters, geom == GEOM_WIDE128,
                         (int)sms, &bn, &csplit);
        const int fs = tuning().conv_csplit;
        if ((fs == 1 || fs == 2 || fs == 4 || fs == 8) && geom != GEOM_TAP16 && bn <= 128)
            csplit = k_iters >= fs ? fs : 1;
    }
    const CUtensorMapSwizzle swz = geom == GEOM_WIDE128 ? CU_TENSOR_MAP_SWIZZLE_128B
                                   : geom == GEOM_WIDE  ? CU_TENSOR_MAP_SWIZZLE_64B
                                                        : CU_TENSOR_MAP_SWIZZLE_NONE;
    CUtensorMap map_a, map_b;
    const bool a_tiled = geom != GEOM_TAP16 && conv_is_plain_matrix(a);
    if (a_tiled) {
        // a pointwise convolution reads the activation as the matrix [N*H*W][IC]: a tiled
        // map, 128 rows per box (rows past the end are filled with zeros)
        cuuint64_t dims[2] = {(cuuint64_t)a.ic, (cuuint64_t)a.m};
        cuuint64_t strides[1] = {(cuuint64_t)a.ic};
        cuuint32_t box[2] = {(cuuint32_t)chans, (cuuint32_t)kBM};
        cuuint32_t estr[2] = {1, 1};
        CUresult r = api.tiled(
                &map_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)src, dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            return set_error(ST_RUNTIME, "cuTensorMapEncodeTiled(activation) failed: %d", (int)r);
    } else {
        // (a small activation is described with the images of readable memory behind it)
        const int images = descriptor_images(a, src);
        if (images == 0)
            return set_error(ST_INVALID_LAYOUT, "activation below 128 KiB outside a registered range");
        cuuint64_t dims[4] = {(cuuint64_t)a.ic, (cuuint64_t)a.iw, (cuuint64_t)a.ih,
                              (cuuint64_t)images};
        cuuint64_t strides[3] = {(cuuint64_t)a.ic, (cuuint64_t)a.iw * a.ic,
                                 (cuuint64_t)a.ih * a.iw * a.ic};
        // bounding box of the first-tap positions: from -pad to the last output's position
        int lower[2] = {-a.pw, -a.ph};
        int upper[2] = {(a.ow - 1) * a.sw - a.pw - (a.iw - 1), (a.oh - 1) * a.sh - a.ph - (a.ih - 1)};
        cuuint32_t estr[4] = {1, (cuuint32_t)a.sw, (cuuint32_t)a.sh, 1};
        CUresult r = api.im2col(
                &map_a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, (void*)src, dims, strides, lower, upper,
                chans, kBM, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            return set_error(ST_RUNTIME, "cuTensorMapEncodeIm2col failed: %d", (int)r);
    }
    {
        const cuuint64_t k_total = (cuuint64_t)taps * a.ic;
        cuuint64_t dims[2] = {k_total, (cuuint64_t)a.oc};
        cuuint64_t strides[1] = {k_total};
        cuuint32_t box[2] = {(cuuint32_t)chans, (cuuint32_t)bn};
        cuuint32_t estr[2] = {1, 1};
        CUresult r = api.tiled(
                &map_b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)flt, dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            return set_error(ST_RUNTIME, "cuTensorMapEncodeTiled failed: %d", (int)r);
    }

    UmmaConvParams p;
    p.m_total = a.m;
    p.oc = a.oc;
    p.oh = a.oh;
    p.ow = a.ow;
    p.cblocks = geom == GEOM_TAP16 ? 1 : (a.ic + chans - 1) / chans;
    p.tap_step = a.ic - (p.cblocks - 1) * chans;
    p.taps_w = a.kw;
    p.k_iters = geom == GEOM_TAP16 ? taps / 4 : taps * p.cblocks;
    p.sh = a.sh;
    p.sw = a.sw;
    p.base_h = -a.ph;
    p.base_w = -a.pw;
    p.dh = a.dh;
    p.dw = a.dw;
    p.m_tiles = (a.m - 1) / kBM + 1;
    p.n_tiles = (a.oc + bn - 1) / bn;
    p.a_tiled = a_tiled ? 1 : 0;
    fill_epilogue(a, bias, flt_scales, &p.ep);
    if (tuning().debug)
        fprintf(stderr, "%s: scales %g %g %g act %d z_mode %d verified requant: %d ops, %g + %.9g, short residual %g %g\n", "conv_umma",
                a.s_src, a.s_flt, a.s_dst, a.act, p.ep.z_mode, p.ep.fast_ops, p.ep.fast_mul, p.ep.fast_add,
                p.ep.z_fast_a,
                p.ep.z_fast_b);
    p.dst = dst;
    p.status = device_status_word(st);
    p.wait_cycles = a.test_wait_cycles > 0 ? a.test_wait_cycles : kWaitCycles;
    p.skip_step = a.test_wait_cycles > 0 ? a.test_skip_step : -1;
    if (!p.status)
        return ST_MALLOC;
    p.full_tiles = p.total_items = p.m_tiles * p.n_tiles;
    p.split = 1;
    p.k_per_part = p.k_iters;
    p.slabs = nullptr;
    p.csplit = csplit;
    p.counters = nullptr;
    if (geom == GEOM_WIDE128) {
        if (bn == 256) {
            const SplitPlan sp = plan_split_k(p.m_tiles * p.n_tiles, p.k_iters, sm_count());
            void* scratch = sp.split > 1 ? split_scratch(st) : nullptr;
            if (scratch) {
                p.full_tiles = sp.full_tiles;
                p.split = sp.split;
                p.k_per_part = sp.k_per_part;
                p.total_items = sp.total_items;
                p.counters = (unsigned*)scratch;
                p.slabs = (int4*)((uint8_t*)scratch + kCounterBytes);
                return launch_form<256, GEOM_WIDE128, true>(map_a, map_b, p, st);
            }
            return launch_kernel<256, GEOM_WIDE128>(map_a, map_b, p, st);
        }
        return bn == 64 ? launch_kernel<64, GEOM_WIDE128>(map_a, map_b, p, st)
                        : launch_kernel<128, GEOM_WIDE128>(map_a, map_b, p, st);
    }
    if (geom == GEOM_WIDE)
        return bn == 64 ? launch_kernel<64, GEOM_WIDE>(map_a, map_b, p, st)
                        : launch_kernel<128, GEOM_WIDE>(map_a, map_b, p, st);
    return bn == 64 ? launch_form<64, GEOM_TAP16>(map_a, map_b, p, st)
                    : launch_form<128, GEOM_TAP16>(map_a, map_b, p, st);
}

int launch_conv_umma(
        const ConvArgs& a, const int8_t* src, const int8_t* flt, const int32_t* bias,
        const float* flt_scales, int8_t* dst, cudaStream_t st) {
    return launch_conv_umma_geom(a, GEOM_WIDE, src, flt, bias, flt_scales, dst, st);
}

}  // namespace mb200
