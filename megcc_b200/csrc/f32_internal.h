// Internal declarations of the fp32 path (conv_f32.cu, f32_ops.cu, f32_abi.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>
#include <string.h>

#include <cuda.h>

#include "../../include/megcc_b200.h"
#include "internal.h"

namespace mb200 {

// Everything an fp32 conv kernel needs, by value. Pitches are in floats.
struct ConvF32Args {
    int n, ic, ih, iw, oc, oh, ow;
    int kh, kw, sh, sw, ph, pw, groups;
    int m;    // n * oh * ow
    int act;  // MB200_F32_*
    long long src_pitch;  // floats between consecutive pixels of src (>= ic)
    long long dst_pitch;  // ... of dst (>= oc): lets a conv write its slice of a concat buffer
    long long z_pitch;    // ... of the optional residual operand
    int forms;       // fp16 planes that the packed filter may hold (F32Forms)
    bool tf32_only;  // not the kernels that use them
};
// A caller of the C ABI packs a filter for every kernel; a network knows which one will run.
enum F32Forms : int { F32_HALF_PLANES = 1, F32_PATCH_PLANES = 2, F32_ALL_PLANES = 3 };

int conv_f32_padded_ic(int ic);
long long conv_f32_tile_clocks(const ConvF32Args& a, int bn);
// does the packed filter begin with the two tf32 planes (else: plain K-major)?
bool conv_f32_split_planes(const ConvF32Args& a);
int conv_f32_forms(const ConvF32Args& a);
size_t conv_f32_split_filter_floats(const ConvF32Args& a);
// fp16 planes for the wide layers (conv_f32_half.cu), behind the tf32 planes of the filters that have them
bool conv_f32_half_planes(const ConvF32Args& a);
size_t conv_f32_half_filter_floats(const ConvF32Args& a);
int launch_conv_f32_pack_filter_half(
        const ConvF32Args& a, const float* flt_oihw, float* out, cudaStream_t st);
int launch_matmul_f32_pack_half(int k, int n, const float* b, float* out, cudaStream_t st);
// 3x3, stride 1, padding 1 from halo patches (conv_f32_patch.cu)
bool conv_f32_patch_planes(const ConvF32Args& a);
bool conv_f32_patch_shape(const ConvF32Args& a);
bool conv_f32_patch_pays(const ConvF32Args& a);
size_t conv_f32_patch_filter_floats(const ConvF32Args& a);
size_t conv_f32_patch_words_at(const ConvF32Args& a);
int launch_conv_f32_pack_filter_patch(
        const ConvF32Args& a, const float* flt_oihw, float* out, cudaStream_t st);
int launch_conv_f32_patch(
        const ConvF32Args& a, const float* src, const float* planes, const float* weights, const float* bias,
        const float* z, float* dst, cudaStream_t st);
size_t matmul_f32_scratch_floats(const ConvF32Args& a, const float* src);
int launch_matmul_f32(
        ConvF32Args a, const float* src, const float* b, float* c, float* scratch, cudaStream_t st);
int launch_conv_f32_half(
        const ConvF32Args& a, const CUtensorMap& map_a, bool a_tiled, const float* src, const float* planes,
        const float* weights, bool weights_raw, const float* bias, const float* z, float* dst, cudaStream_t st);
bool conv_f32_umma_supported(const ConvF32Args& a, const float* src, const float* dst);
// the packed filter of a 1x1 ConvBias from [K][N]
int launch_matmul_f32_pack_b(const ConvF32Args& a, const float* b, float* out, cudaStream_t st);
int launch_conv_f32_pack_filter_split(
        const ConvF32Args& a, const float* flt_oihw, float* out, cudaStream_t st);
int launch_conv_f32_pack_filter_plain(
        const ConvF32Args& a, const float* flt_oihw, float* out, cudaStream_t st);
// [K][N] -> the planes of the 1x1 filter [N][K]
int launch_matmul_f32_pack_split(int k, int n, const float* b, float* out, cudaStream_t st);
int launch_conv_f32_direct(
        const ConvF32Args& a, const float* src, const float* flt_packed, const float* bias,
        const float* z, float* dst, cudaStream_t st);
int launch_conv_f32_umma(
        const ConvF32Args& a, const float* src, const float* flt_split, const float* bias,
        const float* z, float* dst, cudaStream_t st);

int launch_elemwise_f32(
        int mode, const float* a, const float* b, float* dst, size_t nr_elem, cudaStream_t st);
// (pitches: floats between consecutive pixels; concat: null for dense inputs, an input that lies
// in its place of dst already is left alone)
int launch_concat_f32(
        const float* const* srcs, const int* channels, const long long* pitches, int nr, float* dst,
        size_t pixels, cudaStream_t st);
int launch_resize_nearest_f32(
        const float* src, float* dst, int n, int c, int ih, int iw, int oh, int ow,
        long long src_pitch, long long dst_pitch, cudaStream_t st);
int launch_pooling_f32(
        const float* src, float* dst, int mode, int n, int c, int ih, int iw, int wh, int ww,
        int sh, int sw, int ph, int pw, long long src_pitch, long long dst_pitch, cudaStream_t st);
// mb200_conv_bias_f32_nhwc over operands that are slices of wider pixels (0: dense)
int conv_bias_f32_pitched(
        const mb200_conv_f32_param* p, const float* src, long long src_pitch,
        const float* flt_packed, const float* bias, const float* z, long long z_pitch, float* dst,
        long long dst_pitch, int algo, int forms, bool tf32_only, cudaStream_t st);
// the forms that such a ConvBias makes use of, and its filter packed in them
int conv_f32_forms(const mb200_conv_f32_param* p);
size_t conv_f32_packed_bytes(const mb200_conv_f32_param* p, int forms);
int conv_f32_pack(
        const mb200_conv_f32_param* p, int forms, const float* flt_oihw, float* flt_packed, cudaStream_t st);
// Has a packed filter weights that its fp16 planes do not hold (conv_f32_split.cuh)? Its channel words tell:
// where they are (null: it has none), and how many.
const float* conv_f32_filter_words(const mb200_conv_f32_param* p, int forms, const float* flt_packed, int* count);
constexpr uint32_t kWideChannel = 0x80000000u;  // in a channel word
const float* conv_f32_channel_words(const ConvF32Args& a, const float* flt_packed);
int launch_focus_f32(
        const float* src_nchw, float* dst_nhwc, int n, int c, int h, int w, int c_out,
        cudaStream_t st);
int launch_transpose_f32(
        const float* src, float* dst, int batch, int rows, int cols, cudaStream_t st);

}  // namespace mb200
