// Launch of one instantiation of the tensor-core stencil.
#pragma once

#include <algorithm>

#include "launch.h"
#include "mma8.cuh"
#include "mma8.h"
#include "resident.cuh"

namespace kcv {

constexpr int kMma8MaxSmem = 232448 - 2560;  // per CTA, static shared memory aside
static_assert(sizeof(Mma8Taps) + sizeof(Mma8Job) + 16 <= 2560, "");

// CTAs of the kernel on an SM: its register limit (cached) and `dynamic` and
// `fixed` bytes of shared memory.
template <auto Kern>
cudaError_t mma8_resident(int dynamic, int fixed, int *per_sm) {
  int by_regs = 0;
  const cudaError_t e = resident_by_registers<Kern>(kMma8Threads, kMma8MaxSmem, &by_regs);
  if (e != cudaSuccess) return e;
  *per_sm = std::max(1, std::min(by_regs, 233472 / (dynamic + fixed + 1024)));
  return cudaSuccess;
}

template <int NK, int NB, int NA, int MT, int W, int EPI>
cudaError_t launch_mma8_inst(const Mma8Job &j, int sm_count, cudaStream_t stream) {
  int per_sm = 0;
  const cudaError_t e = mma8_resident<mma8_kernel<NK, NB, NA, MT, W, EPI>>(j.smem_bytes, sizeof(Mma8Taps), &per_sm);
  if (e != cudaSuccess) return e;
  const long tiles = static_cast<long>(j.tiles_x) * j.tiles_y;
  const long grid = std::min<long>(tiles, static_cast<long>(per_sm) * sm_count);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(grid));
  cfg.blockDim = dim3(kMma8Threads);
  cfg.dynamicSmemBytes = j.smem_bytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, mma8_kernel<NK, NB, NA, MT, W, EPI>, j);
}

template <int NK, int NB, int NA, int MT, int W, int EPI>
cudaError_t launch_mma8_batch_inst(const Mma8Batch &b, int sm_count, cudaStream_t stream) {
  int per_sm = 0;
  const cudaError_t e = mma8_resident<mma8_batch_kernel<NK, NB, NA, MT, W, EPI>>(
      b.smem_bytes, sizeof(Mma8Taps) + sizeof(Mma8Job) + 16, &per_sm);
  if (e != cudaSuccess) return e;
  const int grid = std::min(b.tiles, per_sm * sm_count);
  // Runs of tiles share one weight table and one pipeline: about six per CTA.
  const int chunk = std::max(1, std::min(16, b.tiles / (6 * grid)));
  mma8_batch_kernel<NK, NB, NA, MT, W, EPI>
      <<<grid, kMma8Threads, b.smem_bytes, stream>>>(b.jobs, b.ends, b.n, chunk, b.next);
  return cudaGetLastError();
}

// The tile sizes of mma8_job: 64 or 32 rows x 256 bytes; batches: 64 rows.
template <int NK, int NB, int NA, int EPI>
cudaError_t launch_mma8_tiled(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream) {
  if (batch) return launch_mma8_batch_inst<NK, NB, NA, 4, 256, EPI>(*batch, sm_count, stream);
  return j.mt == 2 ? launch_mma8_inst<NK, NB, NA, 2, 256, EPI>(j, sm_count, stream)
                   : launch_mma8_inst<NK, NB, NA, 4, 256, EPI>(j, sm_count, stream);
}

}  // namespace kcv
