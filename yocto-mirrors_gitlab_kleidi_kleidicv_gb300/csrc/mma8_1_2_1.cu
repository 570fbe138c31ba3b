// Tensor-core stencil: 3 to 9 taps, horizontal windows of 2 and 1 blocks.
#include "mma8_launch.cuh"

namespace kcv {

cudaError_t launch_mma8_1_2_1(const Mma8Job &j, const Mma8Batch *batch, int sm_count,
                             cudaStream_t stream) {
  return launch_mma8_tiled<1, 2, 1, kEpiRound>(j, batch, sm_count, stream);
}

}  // namespace kcv
