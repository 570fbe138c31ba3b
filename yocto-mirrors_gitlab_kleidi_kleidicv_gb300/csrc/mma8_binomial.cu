// Tensor-core stencil: the binomial kernels of sizes 3 and 5.
#include "mma8_launch.cuh"

namespace kcv {

cudaError_t launch_mma8_binomial(const Mma8Job &j, const Mma8Batch *batch, int sm_count,
                                 cudaStream_t stream) {
  return j.na == 1 ? launch_mma8_tiled<1, 2, 1, kEpiBinomial>(j, batch, sm_count, stream)
                   : launch_mma8_tiled<1, 2, 2, kEpiBinomial>(j, batch, sm_count, stream);
}

}  // namespace kcv
