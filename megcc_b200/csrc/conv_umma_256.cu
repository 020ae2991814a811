// conv_umma_kernel with 256-column tiles
#include "conv_umma_kernel.cuh"

namespace mb200 {
namespace umma_conv {
template int launch_kernel<256, GEOM_WIDE128>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
template int launch_form<256, GEOM_WIDE128, true>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
}  // namespace umma_conv
}  // namespace mb200
