// Sobel 3x3 derivatives, u8 in, s16 out (sm_103a):
// kleidicv_sobel_3x3_{horizontal,vertical}_s16_u8 (kleidicv/src/filters/
// sobel_neon.cpp:12-196; the only border is REPLICATE).
//
// A thread computes 8 neighbouring elements (16 destination bytes) of four
// rows from registers: for each of the six source rows it loads the aligned
// words around its 8 + 2C bytes, shifts them into place and spreads the bytes;
// d/dx is 1 2 1 down the columns of x[e + C] - x[e - C], d/dy the difference two
// rows apart of 1 2 1 along the row.  Threads whose words would leave the row
// gather border-mapped bytes instead.  No shared memory and no barrier: a
// derivative of a camera frame is one short wave of warps that wait for their
// loads (7.9 of 13 cycles per instruction), and the tiled stencil's ring put its
// set-up before them (1920x1080x1 d/dx 6.5 -> 4.1 us).
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "launch.h"
#include "ptx.cuh"

namespace kcv {
namespace {

constexpr int kSobelThreads = 128;
constexpr int kSobelElems = 8;  // elements of a thread in a row
constexpr int kSobelRows = 4;   // and its rows

constexpr int window_words(int c) { return (kSobelElems + 2 * c + 3) / 4; }

struct SobelJob {
  const uint8_t *src;
  uint8_t *dst;
  int64_t src_stride, dst_stride;
  int32_t w, h, wc, groups;  // groups: threads of a row
};

// The bytes [e0 - C, e0 + 8 + C) of a row.
template <int C>
__device__ __forceinline__ void load_window(const SobelJob &j, const uint8_t *row, int e0, bool inner,
                                            int (&x)[kSobelElems + 2 * C]) {
  constexpr int N = kSobelElems + 2 * C, NW = window_words(C);
  if (inner) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(row + e0 - C);
    const uint32_t *p = reinterpret_cast<const uint32_t *>(a & ~uintptr_t{3});
    const int sh = static_cast<int>(a & 3) * 8;
    uint32_t w[NW + 1];
#pragma unroll
    for (int k = 0; k <= NW; ++k) w[k] = ld_src(p + k);
#pragma unroll
    for (int k = 0; k < NW; ++k) {
      const uint32_t v = __funnelshift_r(w[k], w[k + 1], sh);
#pragma unroll
      for (int b = 0; b < 4; ++b)
        if (4 * k + b < N) x[4 * k + b] = static_cast<int>(__byte_perm(v, 0u, 0x4440 + b));
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int e = e0 - C + i, ch = (e + 4 * C) % C;  // e >= -C
      const int lo = max(e, ch), hi = j.wc - C + ch;     // the first and last pixel's element
      x[i] = ld_src(row + min(lo, hi));
    }
  }
}

template <int C, bool DX>
__global__ void __launch_bounds__(kSobelThreads) sobel_kernel(const __grid_constant__ SobelJob j) {
  launch_dependents();
  grid_dependency_wait();  // the source may be the previous call's output
  const int group = blockIdx.x * kSobelThreads + threadIdx.x;
  if (group >= j.groups) return;
  const int e0 = group * kSobelElems;
  // The words read for the window, from up to 3 bytes before it on, lie in the row.
  const bool inner = e0 >= C + 3 && e0 - C + 4 * (window_words(C) + 1) <= j.wc;
  const uintptr_t al = reinterpret_cast<uintptr_t>(j.dst) | static_cast<uintptr_t>(j.dst_stride);
  const int n = min(kSobelElems, j.wc - e0);
  // Row blocks loop over the grid's y extent, which the hardware caps at 65535.
  for (long yb = blockIdx.y; yb * kSobelRows < j.h; yb += gridDim.y) {
    const int y0 = static_cast<int>(yb * kSobelRows);
    int s[kSobelRows + 2][kSobelElems];  // along each source row: difference (d/dx) or 1 2 1 (d/dy)
#pragma unroll
    for (int r = 0; r < kSobelRows + 2; ++r) {
      const int y = min(max(y0 + r - 1, 0), j.h - 1);
      int x[kSobelElems + 2 * C];
      load_window<C>(j, j.src + static_cast<int64_t>(y) * j.src_stride, e0, inner, x);
#pragma unroll
      for (int i = 0; i < kSobelElems; ++i)
        s[r][i] = DX ? x[i + 2 * C] - x[i] : x[i] + 2 * x[i + C] + x[i + 2 * C];
    }
#pragma unroll
    for (int r = 0; r < kSobelRows; ++r) {
      if (y0 + r >= j.h) break;
      uint32_t o[kSobelElems / 2];
#pragma unroll
      for (int i = 0; i < kSobelElems; i += 2) {
        int v[2];
#pragma unroll
        for (int k = 0; k < 2; ++k)
          v[k] = DX ? s[r][i + k] + 2 * s[r + 1][i + k] + s[r + 2][i + k] : s[r + 2][i + k] - s[r][i + k];
        o[i / 2] = __byte_perm(static_cast<uint32_t>(v[0]), static_cast<uint32_t>(v[1]), 0x5410);
      }
      uint8_t *d = j.dst + static_cast<int64_t>(y0 + r) * j.dst_stride + 2 * e0;
      if (n == kSobelElems && (al & 15) == 0) {
        *reinterpret_cast<uint4 *>(d) = make_uint4(o[0], o[1], o[2], o[3]);
      } else if (n == kSobelElems && (al & 3) == 0) {
#pragma unroll
        for (int k = 0; k < 4; ++k) reinterpret_cast<uint32_t *>(d)[k] = o[k];
      } else {
#pragma unroll
        for (int k = 0; k < kSobelElems; ++k)
          if (k < n) reinterpret_cast<uint16_t *>(d)[k] = static_cast<uint16_t>(o[k / 2] >> (16 * (k & 1)));
      }
    }
  }
}

template <int C>
cudaError_t launch_c(const SobelJob &j, bool dx, cudaStream_t stream) {
  const int row_blocks = (j.h + kSobelRows - 1) / kSobelRows;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>((j.groups + kSobelThreads - 1) / kSobelThreads),
                     static_cast<unsigned>(std::min(row_blocks, 65535)));
  cfg.blockDim = dim3(kSobelThreads);
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return dx ? cudaLaunchKernelEx(&cfg, sobel_kernel<C, true>, j) : cudaLaunchKernelEx(&cfg, sobel_kernel<C, false>, j);
}

}  // namespace

bool sobel_eligible(const FilterJob &f) {
  if (f.mode != MODE_SOBEL_X && f.mode != MODE_SOBEL_Y) return false;
  const uintptr_t src = reinterpret_cast<uintptr_t>(f.src) | static_cast<uintptr_t>(f.src_stride);
  const uintptr_t dst = reinterpret_cast<uintptr_t>(f.dst) | static_cast<uintptr_t>(f.dst_stride);
  if (dst & 1) return false;
  // The tiled stencil keeps larger images whose rows TMA can load and 16-byte
  // stores can write.  d/dx, tiled against here: 160x120x1 6.8 / 2.8 us,
  // 1920x1080x1 6.5 / 4.1 us, 1920x1080x3 9.1 / 9.4 us, 3840x2160x4 22.9 / 38.0 us;
  // unaligned 1921x1081x1 46 / 11.5 us, 3841x2160x4 445 / 41 us.
  return ((src | dst) & 15) != 0 || static_cast<long>(f.width) * f.channels * f.height <= 4L << 20;
}

cudaError_t launch_sobel(const FilterJob &f, cudaStream_t stream) {
  SobelJob j{f.src, f.dst, f.src_stride, f.dst_stride, f.width, f.height, f.width * f.channels, 0};
  j.groups = (j.wc + kSobelElems - 1) / kSobelElems;
  const bool dx = f.mode == MODE_SOBEL_X;
  switch (f.channels) {
    case 1: return launch_c<1>(j, dx, stream);
    case 2: return launch_c<2>(j, dx, stream);
    case 3: return launch_c<3>(j, dx, stream);
    case 4: return launch_c<4>(j, dx, stream);
  }
  return cudaErrorInvalidValue;
}

}  // namespace kcv
