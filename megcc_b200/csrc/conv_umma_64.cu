// conv_umma_kernel with 64-column tiles
#include "conv_umma_kernel.cuh"

namespace mb200 {
namespace umma_conv {
template int launch_kernel<64, GEOM_WIDE>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
template int launch_kernel<64, GEOM_WIDE128>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
template int launch_form<64, GEOM_TAP16>(
        const CUtensorMap&, const CUtensorMap&, const UmmaConvParams&, cudaStream_t);
template int umma_clusters<64, GEOM_WIDE>(int);
template int umma_clusters<64, GEOM_WIDE128>(int);
}  // namespace umma_conv
}  // namespace mb200
