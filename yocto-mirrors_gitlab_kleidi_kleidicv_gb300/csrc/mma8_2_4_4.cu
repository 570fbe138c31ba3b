// Tensor-core stencil: 11 to 25 taps, horizontal windows of 4 and 4 blocks.
#include "mma8_launch.cuh"

namespace kcv {

cudaError_t launch_mma8_2_4_4(const Mma8Job &j, const Mma8Batch *batch, int sm_count,
                             cudaStream_t stream) {
  return launch_mma8_tiled<2, 4, 4, kEpiRound>(j, batch, sm_count, stream);
}

}  // namespace kcv
