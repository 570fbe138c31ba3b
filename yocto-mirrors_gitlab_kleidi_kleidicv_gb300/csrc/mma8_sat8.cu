// Tensor-core stencil: the u8 separable filter.
#include "mma8_launch.cuh"

namespace kcv {

cudaError_t launch_mma8_sat8(const Mma8Job &j, const Mma8Batch *batch, int sm_count,
                             cudaStream_t stream) {
  return j.na == 1 ? launch_mma8_tiled<1, 2, 1, kEpiSat8>(j, batch, sm_count, stream)
                   : launch_mma8_tiled<1, 2, 2, kEpiSat8>(j, batch, sm_count, stream);
}

}  // namespace kcv
