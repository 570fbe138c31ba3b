// Host interface of the tensor-core u8 stencils (mma8.cuh, mma8*.cu).
#pragma once

#include <cuda_runtime.h>

#include "kcv_job.h"

namespace kcv {

// Fills the job of a fused Gaussian with generated weights, a u8 separable
// filter or a binomial 3x3 or 5x5 of a smaller or unaligned image, or of an
// arbitrary-size Gaussian, tiled for `sm_count` SMs.  False: the call is not of
// these kinds, or (arbitrary sizes) its images overlap, and the job is not
// filled.
bool mma8_job(const FilterJob &f, int sm_count, Mma8Job &j);
bool mma8_job(const GenericJob &g, int sm_count, Mma8Job &j);
cudaError_t launch_mma8(const Mma8Job &j, int sm_count, cudaStream_t stream);

// Batch plans: n jobs of one instantiation in a device table, job k's tiles
// ending at ends[k] (tiles in all), claimed through *next (0 at launch).
struct Mma8Batch {
  const Mma8Job *jobs;
  const int *ends;
  int n, tiles;
  int *next;
  int smem_bytes;
};
// The instantiation a job belongs to in batch plans (0: none; mma8_batch_job
// tiles it for one).
int mma8_batch_key(const Mma8Job &j);
bool mma8_batch_job(const FilterJob &f, Mma8Job &j);
// `rep` is any job of the batch.
cudaError_t launch_mma8_batch(const Mma8Job &rep, const Mma8Batch &b, int sm_count, cudaStream_t stream);

// Instantiations, one translation unit each: <vertical steps>_<horizontal
// steps nb>_<na>, or any number of steps; the u8
// separable filter; the binomial kernels of sizes 3 and 5.
cudaError_t launch_mma8_1_2_1(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_1_2_2(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_1_3_2(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_1_3_3(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_2_2_2(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_2_3_2(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_2_3_3(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_2_4_4(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_2_5_4(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_3_3_3(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_3_4_3(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_2_any(const Mma8Job &j, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_3_any(const Mma8Job &j, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_0_any(const Mma8Job &j, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_binomial(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);
cudaError_t launch_mma8_sat8(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream);

}  // namespace kcv
