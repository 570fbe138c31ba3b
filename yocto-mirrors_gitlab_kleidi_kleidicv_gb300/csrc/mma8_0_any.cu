// Tensor-core stencil: any number of taps, any horizontal window, and the arbitrary-size forms.
#include "mma8_launch.cuh"

namespace kcv {

cudaError_t launch_mma8_0_any(const Mma8Job &j, int sm_count, cudaStream_t stream) {
  return j.epi == kEpiArbitrary ? launch_mma8_inst<0, 0, 0, 4, 256, kEpiArbitrary>(j, sm_count, stream)
                                : launch_mma8_inst<0, 0, 0, 4, 256, kEpiRound>(j, sm_count, stream);
}

}  // namespace kcv
