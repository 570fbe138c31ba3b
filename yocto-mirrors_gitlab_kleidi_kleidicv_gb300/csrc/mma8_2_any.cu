// Tensor-core stencil: 11 to 25 taps, any horizontal window, and the arbitrary-size forms.
#include "mma8_launch.cuh"

namespace kcv {

cudaError_t launch_mma8_2_any(const Mma8Job &j, int sm_count, cudaStream_t stream) {
  return j.epi == kEpiArbitrary ? launch_mma8_inst<2, 0, 0, 4, 256, kEpiArbitrary>(j, sm_count, stream)
                                : launch_mma8_inst<2, 0, 0, 4, 256, kEpiRound>(j, sm_count, stream);
}

}  // namespace kcv
