// extern "C" entry points of the fp32 path declared in include/megcc_b200.h.
#include "f32_internal.h"

using namespace mb200;

namespace {

size_t up256(size_t v) {
    return (v + 255) / 256 * 256;
}

int make_f32_args(const mb200_conv_f32_param* p, long long dst_pitch, ConvF32Args* a) {
    if (!p)
        return set_error(ST_NULL_PTR, "conv param is NULL");
    if (p->n <= 0 || p->ic <= 0 || p->oc <= 0 || p->ih <= 0 || p->iw <= 0 || p->kh <= 0 ||
        p->kw <= 0 || p->stride_h <= 0 || p->stride_w <= 0 || p->pad_h < 0 || p->pad_w < 0 ||
        p->groups <= 0)
        return set_error(ST_INVALID_LAYOUT, "conv param has a non-positive extent");
    if (p->ic % p->groups || p->oc % p->groups)
        return set_error(ST_INVALID_LAYOUT, "channels %d/%d not divisible by groups %d", p->ic,
                         p->oc, p->groups);
    if (p->nonline < 0 || p->nonline > MB200_F32_SILU)
        return set_error(ST_NO_IMPLEMENT, "nonlineMode %d not supported", p->nonline);
    a->n = p->n;
    a->ic = p->ic;
    a->ih = p->ih;
    a->iw = p->iw;
    a->oc = p->oc;
    a->kh = p->kh;
    a->kw = p->kw;
    a->sh = p->stride_h;
    a->sw = p->stride_w;
    a->ph = p->pad_h;
    a->pw = p->pad_w;
    a->groups = p->groups;
    a->oh = out_extent(p->ih, p->kh, p->stride_h, p->pad_h, 1);
    a->ow = out_extent(p->iw, p->kw, p->stride_w, p->pad_w, 1);
    if (a->oh <= 0 || a->ow <= 0)
        return set_error(ST_INVALID_LAYOUT, "filter larger than the padded input");
    const long long m = (long long)p->n * a->oh * a->ow;
    if (m > 0x3fffffffLL)
        return set_error(ST_OUT_OF_RANGE, "too many output pixels");
    a->m = (int)m;
    a->act = p->nonline;
    a->forms = F32_ALL_PLANES;
    a->tf32_only = false;
    a->src_pitch = p->ic;
    a->dst_pitch = dst_pitch > 0 ? dst_pitch : p->oc;
    a->z_pitch = p->oc;
    if (a->dst_pitch < p->oc)
        return set_error(ST_INVALID_LAYOUT, "dst_pitch %lld is below the channel count %d",
                         a->dst_pitch, p->oc);
    return ST_SUCCESS;
}

size_t plain_filter_bytes(const ConvF32Args& a) {
    return up256((size_t)a.oc * (a.ic / a.groups) * a.kh * a.kw * sizeof(float));
}

}  // namespace

namespace mb200 {

int conv_bias_f32_pitched(
        const mb200_conv_f32_param* p, const float* src, long long src_pitch,
        const float* flt_packed, const float* bias, const float* z, long long z_pitch, float* dst,
        long long dst_pitch, int algo, int forms, bool tf32_only, cudaStream_t st) {
    ConvF32Args a{};
    int rc = make_f32_args(p, dst_pitch, &a);
    if (rc)
        return rc;
    if (src_pitch > 0)
        a.src_pitch = src_pitch;
    if (z_pitch > 0)
        a.z_pitch = z_pitch;
    a.forms = forms;
    a.tf32_only = tf32_only;
    if (!src || !flt_packed || !dst)
        return set_error(ST_NULL_PTR, "conv tensor pointer is NULL");
    if (((uintptr_t)src | (uintptr_t)flt_packed | (uintptr_t)dst | (uintptr_t)bias |
         (uintptr_t)z) & 3)
        return set_error(ST_INVALID_LAYOUT, "fp32 operands must be 4-byte aligned");
    const bool umma_ok = conv_f32_umma_supported(a, src, dst) &&
                         (((uintptr_t)flt_packed | (uintptr_t)bias | (uintptr_t)z) & 15) == 0;
    if (algo == MB200_ALGO_UMMA && !umma_ok)
        return set_error(ST_NO_IMPLEMENT,
                         "tensor-core fp32 ConvBias needs a dense filter, ic %% 4 == 0 (with a spatial "
                         "filter ic == 16 or ic >= 32), 16-byte aligned operands and, with a spatial "
                         "filter, >= 128 KiB of readable memory from the input on");
    if (algo == MB200_ALGO_UMMA || (algo == MB200_ALGO_AUTO && umma_ok))
        return launch_conv_f32_umma(a, src, flt_packed, bias, z, dst, st);
    if (algo != MB200_ALGO_AUTO && algo != MB200_ALGO_DIRECT)
        return set_error(ST_OUT_OF_RANGE, "unknown algo %d", algo);
    return launch_conv_f32_direct(a, src, flt_packed, bias, z, dst, st);
}

int conv_f32_forms(const mb200_conv_f32_param* p) {
    ConvF32Args a{};
    return make_f32_args(p, 0, &a) ? 0 : conv_f32_forms(a);
}

size_t conv_f32_packed_bytes(const mb200_conv_f32_param* p, int forms) {
    ConvF32Args a{};
    if (make_f32_args(p, 0, &a))
        return 0;
    a.forms = forms;
    return conv_f32_split_planes(a) ? up256(conv_f32_split_filter_floats(a) * sizeof(float))
                                    : plain_filter_bytes(a);
}

int conv_f32_pack(
        const mb200_conv_f32_param* p, int forms, const float* flt_oihw, float* flt_packed, cudaStream_t st) {
    ConvF32Args a{};
    int rc = make_f32_args(p, 0, &a);
    if (rc)
        return rc;
    a.forms = forms;
    if (!flt_oihw || !flt_packed)
        return set_error(ST_NULL_PTR, "filter pointer is NULL");
    if (((uintptr_t)flt_oihw & 3) || ((uintptr_t)flt_packed & 15))
        return set_error(ST_INVALID_LAYOUT, "filter must be 4-byte, packed filter 16-byte aligned");
    return conv_f32_split_planes(a) ? launch_conv_f32_pack_filter_split(a, flt_oihw, flt_packed, st)
                                    : launch_conv_f32_pack_filter_plain(a, flt_oihw, flt_packed, st);
}

const float* conv_f32_filter_words(
        const mb200_conv_f32_param* p, int forms, const float* flt_packed, int* count) {
    ConvF32Args a{};
    if (make_f32_args(p, 0, &a))
        return nullptr;
    a.forms = forms;
    *count = a.oc;
    return conv_f32_channel_words(a, flt_packed);
}

}  // namespace mb200

extern "C" {

size_t mb200_conv_f32_packed_filter_bytes(const mb200_conv_f32_param* p) {
    return conv_f32_packed_bytes(p, F32_ALL_PLANES);
}

int mb200_conv_f32_pack_filter(
        const mb200_conv_f32_param* p, const float* flt_oihw, float* flt_packed, void* stream) {
    return conv_f32_pack(p, F32_ALL_PLANES, flt_oihw, flt_packed, (cudaStream_t)stream);
}

// (kept, like the workspace arguments, for callers of earlier versions: the operands are split on
// chip, no scratch is used)
size_t mb200_conv_f32_workspace_bytes(const mb200_conv_f32_param*) {
    return 0;
}

int mb200_conv_bias_f32_nhwc(
        const mb200_conv_f32_param* p, const float* src, const float* flt_packed,
        const float* bias, const float* z, float* dst, long long dst_pitch, void*, size_t, int algo,
        void* stream) {
    return conv_bias_f32_pitched(p, src, 0, flt_packed, bias, z, 0, dst, dst_pitch, algo, F32_ALL_PLANES,
                                 false, (cudaStream_t)stream);
}

// ---- fp32 matrix product: a 1x1 ConvBias over M "pixels" with K channels ----
static int matmul_f32_param(int m, int n, int k, mb200_conv_f32_param* p) {
    if (m <= 0 || n <= 0 || k <= 0)
        return set_error(ST_INVALID_LAYOUT, "matmul extents must be positive");
    memset(p, 0, sizeof(*p));
    p->n = m;
    p->ic = k;
    p->ih = p->iw = 1;
    p->oc = n;
    p->kh = p->kw = 1;
    p->stride_h = p->stride_w = 1;
    p->groups = 1;
    p->nonline = MB200_F32_IDENTITY;
    return ST_SUCCESS;
}

size_t mb200_matmul_f32_packed_b_bytes(int k, int n) {
    mb200_conv_f32_param p;
    if (matmul_f32_param(1, n, k, &p))
        return 0;
    return mb200_conv_f32_packed_filter_bytes(&p);
}

int mb200_matmul_f32_pack_b(int k, int n, const float* b, float* b_packed, void* stream) {
    mb200_conv_f32_param p;
    int rc = matmul_f32_param(1, n, k, &p);
    if (rc)
        return rc;
    if (!b || !b_packed)
        return set_error(ST_NULL_PTR, "matmul operand pointer is NULL");
    if (((uintptr_t)b & 3) || ((uintptr_t)b_packed & 15))
        return set_error(ST_INVALID_LAYOUT, "B must be 4-byte, the packed B 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    ConvF32Args a{};
    if ((rc = make_f32_args(&p, 0, &a)))
        return rc;
    // [K][N] row-major -> [N][K], the K-major filter of a 1x1 conv (or its planes)
    return conv_f32_split_planes(a) ? launch_matmul_f32_pack_b(a, b, b_packed, st)
                                    : launch_transpose_f32(b, b_packed, 1, k, n, st);
}

size_t mb200_matmul_f32_workspace_bytes(int, int) {
    return 0;
}

int mb200_matmul_f32(
        int m, int n, int k, const float* a, const float* b_packed, float* c, void*, size_t,
        void* stream) {
    mb200_conv_f32_param p;
    int rc = matmul_f32_param(m, n, k, &p);
    if (rc)
        return rc;
    if (!a || !b_packed || !c)
        return set_error(ST_NULL_PTR, "matmul operand pointer is NULL");
    return mb200_conv_bias_f32_nhwc(&p, a, b_packed, nullptr, nullptr, c, 0, nullptr, 0,
                                    MB200_ALGO_AUTO, stream);
}

static int product_args(int m, int n, int k, ConvF32Args* a) {
    mb200_conv_f32_param p;
    const int rc = matmul_f32_param(m, n, k, &p);
    return rc ? rc : make_f32_args(&p, 0, a);
}

size_t mb200_matmul_f32_scratch_bytes_for(int m, int n, int k, const float* a) {
    ConvF32Args args{};
    return product_args(m, n, k, &args) ? 0 : up256(matmul_f32_scratch_floats(args, a) * sizeof(float));
}

size_t mb200_matmul_f32_scratch_bytes(int m, int n, int k) {
    return mb200_matmul_f32_scratch_bytes_for(m, n, k, (const float*)4);  // (an address that needs the copy)
}

int mb200_matmul_f32_product(
        int m, int n, int k, const float* a, const float* b, float* c, void* scratch,
        size_t scratch_bytes, void* stream) {
    ConvF32Args args{};
    const int rc = product_args(m, n, k, &args);
    if (rc)
        return rc;
    if (!a || !b || !c || !scratch)
        return set_error(ST_NULL_PTR, "matmul operand or scratch pointer is NULL");
    if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 3)
        return set_error(ST_INVALID_LAYOUT, "fp32 operands must be 4-byte aligned");
    if ((uintptr_t)scratch & 15)
        return set_error(ST_INVALID_LAYOUT, "scratch must be 16-byte aligned");
    if (scratch_bytes < mb200_matmul_f32_scratch_bytes_for(m, n, k, a))
        return set_error(ST_OUT_OF_RANGE, "scratch of %zu bytes is too small", scratch_bytes);
    cudaStream_t st = (cudaStream_t)stream;
    if (((uintptr_t)c & 15) == 0)
        return launch_matmul_f32(args, a, b, c, (float*)scratch, st);
    // (a result that no vector store reaches: the general kernel, which reads the first planes only)
    const int pack = conv_f32_split_planes(args)
                             ? launch_matmul_f32_pack_split(k, n, b, (float*)scratch, st)
                             : launch_transpose_f32(b, (float*)scratch, 1, k, n, st);
    return pack ? pack
                : launch_conv_f32_direct(args, a, (const float*)scratch, nullptr, nullptr, c, st);
}

int mb200_elemwise_f32(
        int mode, const float* a, const float* b, float* dst, size_t nr_elem, void* stream) {
    const bool unary = mode >= MB200_ELEM_RELU && mode <= MB200_ELEM_EXP;
    const bool binary = mode >= MB200_ELEM_ADD && mode <= MB200_ELEM_FUSE_ADD_RELU;
    if (!unary && !binary)
        return set_error(ST_NO_IMPLEMENT, "elemwise mode %d not supported", mode);
    if (!a || !dst || (binary && !b))
        return set_error(ST_NULL_PTR, "elemwise tensor pointer is NULL");
    if (((uintptr_t)a | (uintptr_t)b | (uintptr_t)dst) & 3)
        return set_error(ST_INVALID_LAYOUT, "fp32 operands must be 4-byte aligned");
    if (nr_elem == 0)
        return ST_SUCCESS;
    return launch_elemwise_f32(mode, a, binary ? b : a, dst, nr_elem, (cudaStream_t)stream);
}

int mb200_concat_f32_nhwc(
        const float* const* srcs, const int* channels, int nr_inputs, float* dst, size_t pixels,
        void* stream) {
    if (!srcs || !channels || !dst)
        return set_error(ST_NULL_PTR, "concat pointer is NULL");
    if (pixels == 0)
        return ST_SUCCESS;
    return launch_concat_f32(srcs, channels, nullptr, nr_inputs, dst, pixels, (cudaStream_t)stream);
}

int mb200_resize_nearest_f32_nhwc(
        const float* src, float* dst, int n, int c, int ih, int iw, int oh, int ow, void* stream) {
    if (!src || !dst)
        return set_error(ST_NULL_PTR, "resize tensor pointer is NULL");
    if (n <= 0 || c <= 0 || ih <= 0 || iw <= 0 || oh <= 0 || ow <= 0)
        return set_error(ST_INVALID_LAYOUT, "resize extents must be positive");
    return launch_resize_nearest_f32(src, dst, n, c, ih, iw, oh, ow, c, c, (cudaStream_t)stream);
}

int mb200_pooling_f32_nhwc(
        const float* src, float* dst, int mode, int n, int c, int ih, int iw, int window_h,
        int window_w, int stride_h, int stride_w, int pad_h, int pad_w, void* stream) {
    if (!src || !dst)
        return set_error(ST_NULL_PTR, "pooling tensor pointer is NULL");
    if (mode < 0 || mode > 2)
        return set_error(ST_NO_IMPLEMENT, "pooling mode %d not supported", mode);
    if (n <= 0 || c <= 0 || ih <= 0 || iw <= 0 || window_h <= 0 || window_w <= 0 ||
        stride_h <= 0 || stride_w <= 0 || pad_h < 0 || pad_w < 0 ||
        ih + 2 * pad_h < window_h || iw + 2 * pad_w < window_w || pad_h >= window_h ||
        pad_w >= window_w)
        return set_error(ST_INVALID_LAYOUT, "pooling extents are invalid");
    return launch_pooling_f32(src, dst, mode, n, c, ih, iw, window_h, window_w, stride_h,
                              stride_w, pad_h, pad_w, c, c, (cudaStream_t)stream);
}

int mb200_focus_f32(
        const float* src_nchw, float* dst_nhwc, int n, int c, int h, int w, int c_out,
        void* stream) {
    if (!src_nchw || !dst_nhwc)
        return set_error(ST_NULL_PTR, "focus tensor pointer is NULL");
    if (n <= 0 || c <= 0 || h <= 0 || w <= 0 || (h & 1) || (w & 1) || c_out < 4 * c)
        return set_error(ST_INVALID_LAYOUT, "focus needs even extents and c_out >= 4 * c");
    return launch_focus_f32(src_nchw, dst_nhwc, n, c, h, w, c_out, (cudaStream_t)stream);
}

int mb200_relayout_nchw_to_nhwc_f32(
        const float* src, float* dst, int n, int c, int h, int w, void* stream) {
    if (!src || !dst)
        return set_error(ST_NULL_PTR, "relayout tensor pointer is NULL");
    return launch_transpose_f32(src, dst, n, c, h * w, (cudaStream_t)stream);
}

int mb200_relayout_nhwc_to_nchw_f32(
        const float* src, float* dst, int n, int c, int h, int w, void* stream) {
    if (!src || !dst)
        return set_error(ST_NULL_PTR, "relayout tensor pointer is NULL");
    return launch_transpose_f32(src, dst, n, h * w, c, (cudaStream_t)stream);
}

}  // extern "C"
