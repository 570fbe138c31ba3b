// Median blur on the GPU: kleidicv_median_blur_{s8,u8,u16,s16,u32,s32,f32}
// (kleidicv/src/filters/median_blur_api.cpp, validation in
// kleidicv/include/kleidicv/filters/median_blur.h:148-193).  The result is the
// median of the border-mapped K x K window of every element, which is unique,
// so any exact selection reproduces the reference's sorting networks
// (K = 3, 5, 7) and histograms (u8, K = 9..255).
//
//  * K <= 7: order-preserving unsigned keys, two 16-bit ones per word, through
//    min/max networks that share sorting between neighbouring windows
//    (median3_kernel, median_small_kernel).
//  * u8, K >= 9: Huang's sliding histogram.  A thread owns a run of
//    max(16, K/2) pixels of one row and channel and a 256-bin histogram in
//    shared memory (bins outermost, so the 64 threads of a block hit distinct
//    banks); moving one pixel right removes a column, adds a column and moves
//    the median bin by the count of values that crossed it.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/kleidicv_gpu.h"
#include "host.h"
#include "launch.h"
#include "sepfused.cuh"

namespace kcv {
namespace {

// Order-preserving unsigned keys.  Floats: sign-magnitude to offset binary
// (-0.0 orders just below +0.0).
template <typename T>
struct Key;
template <>
struct Key<uint8_t> {
  __device__ static uint32_t to(uint8_t v) { return v; }
  __device__ static uint8_t from(uint32_t k) { return static_cast<uint8_t>(k); }
};
template <>
struct Key<int8_t> {
  __device__ static uint32_t to(int8_t v) { return static_cast<uint8_t>(v) ^ 0x80u; }
  __device__ static int8_t from(uint32_t k) { return static_cast<int8_t>(k ^ 0x80u); }
};
template <>
struct Key<uint16_t> {
  __device__ static uint32_t to(uint16_t v) { return v; }
  __device__ static uint16_t from(uint32_t k) { return static_cast<uint16_t>(k); }
};
template <>
struct Key<int16_t> {
  __device__ static uint32_t to(int16_t v) { return static_cast<uint16_t>(v) ^ 0x8000u; }
  __device__ static int16_t from(uint32_t k) { return static_cast<int16_t>(k ^ 0x8000u); }
};
template <>
struct Key<uint32_t> {
  __device__ static uint32_t to(uint32_t v) { return v; }
  __device__ static uint32_t from(uint32_t k) { return k; }
};
template <>
struct Key<int32_t> {
  __device__ static uint32_t to(int32_t v) { return static_cast<uint32_t>(v) ^ 0x80000000u; }
  __device__ static int32_t from(uint32_t k) { return static_cast<int32_t>(k ^ 0x80000000u); }
};
template <>
struct Key<float> {
  __device__ static uint32_t to(float v) {
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  }
  __device__ static float from(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
  }
};

// Two elements of at most 16 bits share a word (and its min/max instructions).
template <bool PACKED>
__device__ __forceinline__ uint32_t vmin(uint32_t a, uint32_t b) {
  if constexpr (PACKED) return __vminu2(a, b);
  else return min(a, b);
}
template <bool PACKED>
__device__ __forceinline__ uint32_t vmax(uint32_t a, uint32_t b) {
  if constexpr (PACKED) return __vmaxu2(a, b);
  else return max(a, b);
}
template <bool PACKED>
__device__ __forceinline__ void cex(uint32_t &lo, uint32_t &hi) {
  const uint32_t a = vmin<PACKED>(lo, hi), b = vmax<PACKED>(lo, hi);
  lo = a;
  hi = b;
}

// Compare-exchange lists.  Sorts of K - 1 values (4 and 6: 5 and 12
// exchanges).
template <int N>
struct SortNet;
template <>
struct SortNet<4> {
  static constexpr int n = 5;
  static constexpr int8_t ab[n][2] = {{0, 1}, {2, 3}, {0, 2}, {1, 3}, {1, 2}};
};
template <>
struct SortNet<6> {
  static constexpr int n = 12;
  static constexpr int8_t ab[n][2] = {{0, 5}, {1, 3}, {2, 4}, {1, 2}, {3, 4}, {0, 3},
                                      {2, 5}, {0, 1}, {2, 3}, {4, 5}, {1, 2}, {3, 4}};
};

// The median of a K x K matrix whose rows and columns are sorted: entry (i, j)
// has at least (i + 1)(j + 1) - 1 entries below and (K - i)(K - j) - 1 above
// it, so only those with both products at most (K K + 1) / 2 can be the
// median.  at[] lists them (row, column) as the wires of a selection network
// whose wire `out` ends as the median.  The networks were found by pruning
// sorting networks of the candidates in orders along the matrix's partial
// order, and hold for each of the matrix's C(2K, K) sorted 0-1 patterns (which
// proves them for all inputs); as written only the needed halves of the
// exchanges are computed: 22 and 94 minima and maxima.
template <int K>
struct FinalNet;
template <>
struct FinalNet<5> {
  static constexpr int wires = 13, n = 17, out = 6;
  static constexpr int8_t at[wires][2] = {{1, 2}, {0, 3}, {2, 1}, {3, 0}, {3, 1}, {2, 2}, {4, 0},
                                          {0, 4}, {3, 2}, {1, 4}, {1, 3}, {2, 3}, {4, 1}};
  static constexpr int8_t ab[n][2] = {{0, 1}, {2, 3}, {4, 5}, {6, 7}, {1, 3},  {4, 6}, {5, 7}, {8, 10}, {9, 11},
                                      {5, 6}, {8, 12}, {3, 5}, {5, 6}, {5, 9}, {3, 5}, {6, 8}, {5, 6}};
};
template <>
struct FinalNet<7> {
  static constexpr int wires = 29, n = 61, out = 14;
  static constexpr int8_t at[wires][2] = {{0, 4}, {3, 1}, {1, 3}, {2, 3}, {2, 2}, {4, 0}, {4, 1}, {2, 4}, {1, 4}, {6, 0},
                                      {0, 6}, {5, 0}, {3, 3}, {1, 5}, {5, 1}, {5, 2}, {3, 2}, {6, 1}, {3, 4}, {2, 5},
                                      {4, 2}, {4, 3}, {0, 5}, {3, 5}, {1, 6}, {2, 6}, {6, 2}, {4, 4}, {5, 3}};
  static constexpr int8_t ab[n][2] = {{6, 7}, {8, 9}, {10, 11}, {12, 13}, {26, 27}, {0, 2}, {4, 6}, {8, 10}, {9, 11}, {12, 14},
                                      {13, 15}, {17, 19}, {20, 22}, {21, 23}, {24, 26}, {9, 10}, {13, 14}, {17, 18}, {21, 22}, {1, 5},
                                      {2, 6}, {9, 13}, {10, 14}, {16, 20}, {17, 21}, {18, 22}, {3, 5}, {10, 12}, {11, 13}, {18, 20},
                                      {19, 21}, {5, 6}, {11, 12}, {13, 14}, {17, 18}, {19, 20}, {20, 28}, {5, 9}, {6, 10}, {7, 11},
                                      {20, 24}, {21, 25}, {7, 9}, {10, 12}, {11, 13}, {18, 20}, {19, 21}, {9, 10}, {11, 12}, {17, 18},
                                      {19, 20}, {9, 17}, {10, 18}, {11, 19}, {12, 20}, {12, 16}, {13, 17}, {14, 18}, {11, 13}, {14, 16},
                                      {13, 14}};
};

template <bool PACKED, int N>
__device__ __forceinline__ void sort_net(uint32_t (&a)[N]) {
  static_for<0, SortNet<N>::n>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    constexpr int lo = SortNet<N>::ab[i][0], hi = SortNet<N>::ab[i][1];
    cex<PACKED>(a[lo], a[hi]);
  });
}
// out = the K sorted values s[0..K-2] and x.
template <bool PACKED, int K>
__device__ __forceinline__ void insert(const uint32_t (&s)[K - 1], uint32_t x, uint32_t (&out)[K]) {
  out[0] = vmin<PACKED>(x, s[0]);
#pragma unroll
  for (int i = 1; i < K - 1; ++i) out[i] = vmax<PACKED>(s[i - 1], vmin<PACKED>(x, s[i]));
  out[K - 1] = vmax<PACKED>(x, s[K - 2]);
}

template <bool PACKED>
__device__ __forceinline__ uint32_t med3(uint32_t a, uint32_t b, uint32_t c) {
  return vmax<PACKED>(vmin<PACKED>(a, b), vmin<PACKED>(vmax<PACKED>(a, b), c));
}

// K = 3: a thread computes one element of four rows from registers.  The three
// neighbours of each source row are sorted once and serve the windows of three
// output rows: the median of nine is the median of the largest minimum, the
// median middle and the smallest maximum of the window's rows.  Packed: rows r
// and r + 2 share a word, 12 minima and maxima per element (18 otherwise) where
// selecting from each window took 42.  Measured: u8 1920x1080x1 14.4 -> 7.1 us,
// 160x120x1 4.2 -> 3.8 us; f32 1280x720x3 18.6 -> 10.8 us (the kernel below, at
// K = 3: 8.3, 6.3 and 20.5 us; non-coherent loads, which a source still being
// written rules out, f32 10.0 us, 8 and 16 bits the same).  Bound by issue: 68 % of the slots and half of
// the ALU pipe, 18 % of the load pipe, 74 % of the warps resident.
template <typename T>
__global__ void __launch_bounds__(128) median3_kernel(const uint8_t *src, int64_t src_stride, uint8_t *dst,
                                                      int64_t dst_stride, int w, int h, int c, int border) {
  constexpr bool PACKED = sizeof(T) <= 2;
  constexpr int N = PACKED ? 4 : 6;  // sorted rows
  launch_dependents();
  grid_dependency_wait();  // the source may be the previous call's output
  const int xe = blockIdx.x * blockDim.x + threadIdx.x;  // element index in the row
  if (xe >= w * c) return;
  const int col = xe / c, ch = xe - col * c;
  int at[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) at[d] = map_index(col + d - 1, w, border) * c + ch;
  // Row blocks loop over the grid's y extent, which the hardware caps at 65535.
  for (long yb = blockIdx.y; yb * 4 < h; yb += gridDim.y) {
    const int y0 = static_cast<int>(yb * 4);
    uint32_t key[6][3];
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      const T *row = reinterpret_cast<const T *>(
          src + static_cast<int64_t>(map_index(y0 + r - 1, h, border)) * src_stride);
#pragma unroll
      for (int d = 0; d < 3; ++d) key[r][d] = Key<T>::to(ld_src(row + at[d]));
    }
    uint32_t s[N][3];
#pragma unroll
    for (int r = 0; r < N; ++r) {
#pragma unroll
      for (int d = 0; d < 3; ++d) s[r][d] = PACKED ? key[r][d] | key[r + 2][d] << 16 : key[r][d];
      cex<PACKED>(s[r][0], s[r][1]);
      cex<PACKED>(s[r][1], s[r][2]);
      cex<PACKED>(s[r][0], s[r][1]);
    }
#pragma unroll
    for (int r = 0; r < N - 2; ++r) {
      const uint32_t lo = vmax<PACKED>(vmax<PACKED>(s[r][0], s[r + 1][0]), s[r + 2][0]);
      const uint32_t mid = med3<PACKED>(s[r][1], s[r + 1][1], s[r + 2][1]);
      const uint32_t hi = vmin<PACKED>(vmin<PACKED>(s[r][2], s[r + 1][2]), s[r + 2][2]);
      const uint32_t m = med3<PACKED>(lo, mid, hi);
      auto store = [&](int y, uint32_t k) {
        if (y < h) reinterpret_cast<T *>(dst + static_cast<int64_t>(y) * dst_stride)[xe] = Key<T>::from(k);
      };
      if constexpr (PACKED) {
        store(y0 + r, m & 0xFFFFu);
        store(y0 + r + 2, m >> 16);
      } else {
        store(y0 + r, m);
      }
    }
  }
}

// K = 5, 7: a block stages the border-mapped keys of up to 16 rows x 32 CW
// pixels and their halo in shared memory, planar by channel; a lane then
// computes CW neighbouring pixels of two rows (packed: two more rows, the
// words holding row r and row r + 2).  Windows share their work: the K - 1
// rows that both output rows read are sorted per column once and the row above
// or below inserted; then each rank of the sorted columns is sorted across the
// K - 1 columns that two neighbouring windows share and the outer column
// inserted (entries that cannot be the median are never computed); the
// selection network takes the median of what is left: about 50 half-rate minima
// and maxima per element (packed: two elements) at K = 5, where selecting from
// each window by itself took 330.  Measured (1920x1080x1): u8 K = 5 / 7 49.4 /
// 152 -> 12.1 / 26.5 us, f32 K = 5 49.4 -> 20.0 us; 160x120 K = 5 6.2 -> 3.8 us.
// Few warps and no full pipe: half of the ALU pipe and 40 % of the issue slots
// at 16 % of the warps resident (three blocks of up to 168 registers).  Of a
// warp's 6.3 cycles per instruction 1.8 are fixed waits between dependent
// instructions, 0.7 global loads, 0.6 the ALU pipe, 0.4 shared memory.  Four
// blocks of 128 registers spill: u8 1920x1080x3 K = 5 32.1 -> 28.3 us, but
// 1280x720x1 5.6 -> 7.8 us and u16 1920x1080x1 11.9 -> 13.5 us.
constexpr int median_width(int k) { return k == 7 ? 2 : 4; }  // pixels of a lane
constexpr int median_pitch(int k) { return (32 * median_width(k) + k - 1 + 3) / 4 * 4; }
constexpr int median_group(bool packed) { return packed ? 4 : 2; }  // output rows of a lane
__host__ __device__ constexpr int median_stage_rows(int rows, int k, bool packed) {
  return rows + k - 1 - (packed ? 2 : 0);
}

// Source rows y0 - R .. of the block's columns (and halo) as keys.  A warp
// takes every fourth row, three rows at a time, and issues five loads of each
// before it stores the first; packed keys go to the low half of their row's
// words and the high half of the words two rows above.  C channels from
// channel c0 on, of images of `c`.
template <typename T, int K, int C>
__device__ __forceinline__ void median_stage(uint32_t *stage, const uint8_t *src, int64_t src_stride, int w, int h,
                                             int border, int x0, int y0, int rows, int c, int c0) {
  constexpr bool PACKED = sizeof(T) <= 2;
  constexpr int R = K / 2, P = median_pitch(K), kAhead = 5, kRows = 3;
  const int stage_rows = median_stage_rows(rows, K, PACKED);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = (min(32 * median_width(K), w - x0) + K - 1) * C;
  const bool inner = x0 >= R && x0 - R + n / C <= w;  // no column to map
  for (int row0 = warp; row0 < rows + K - 1; row0 += 4 * kRows) {
    const T *r[kRows];
#pragma unroll
    for (int q = 0; q < kRows; ++q)
      r[q] = reinterpret_cast<const T *>(
          src + static_cast<int64_t>(map_index(y0 - R + row0 + 4 * q, h, border)) * src_stride);
    for (int i0 = lane; i0 < n; i0 += 32 * kAhead) {
      uint32_t v[kRows][kAhead];
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        const int i = i0 + 32 * k;
        if (i >= n) continue;
        const int px = i / C;
        const int at = (inner ? x0 - R + px : map_index(x0 - R + px, w, border)) * (C > 1 ? C : c) + c0 + (i - px * C);
#pragma unroll
        for (int q = 0; q < kRows; ++q) v[q][k] = Key<T>::to(ld_src(r[q] + at));
      }
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        const int i = i0 + 32 * k;
        if (i >= n) continue;
        const int px = i / C;
        uint32_t *d = stage + (i - px * C) * stage_rows * P + px;
#pragma unroll
        for (int q = 0; q < kRows; ++q) {
          const int row = row0 + 4 * q;
          if constexpr (PACKED) {
            if (row < stage_rows) reinterpret_cast<uint16_t *>(d + row * P)[0] = static_cast<uint16_t>(v[q][k]);
            if (row >= 2 && row < stage_rows + 2)
              reinterpret_cast<uint16_t *>(d + (row - 2) * P)[1] = static_cast<uint16_t>(v[q][k]);
          } else {
            if (row < stage_rows) d[row * P] = v[q][k];
          }
        }
      }
    }
  }
}

template <typename T, int K>
__global__ void __launch_bounds__(128)
    median_small_kernel(const uint8_t *src, int64_t src_stride, uint8_t *dst, int64_t dst_stride, int w, int h, int c,
                        int border, int rows) {
  constexpr bool PACKED = sizeof(T) <= 2;
  constexpr int CW = median_width(K), TX = 32 * CW, CC = CW + K - 1;
  constexpr int P = median_pitch(K), GROUP = median_group(PACKED);
  const int stage_rows = median_stage_rows(rows, K, PACKED);
  // All channels in a block, or one per grid layer.
  const int channels = gridDim.z > 1 ? 1 : c, c0 = blockIdx.z;
  extern __shared__ __align__(16) uint32_t median_mem[];
  launch_dependents();
  grid_dependency_wait();  // the source may be the previous call's output
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x0 = blockIdx.x * TX;
  // Row blocks loop over the grid's y extent, which the hardware caps at 65535.
  for (long yb = blockIdx.y; yb * rows < h; yb += gridDim.y) {
    const int y0 = static_cast<int>(yb * rows);
    __syncthreads();  // the last block's reads are done
    switch (channels) {
      case 1: median_stage<T, K, 1>(median_mem, src, src_stride, w, h, border, x0, y0, rows, c, c0); break;
      case 2: median_stage<T, K, 2>(median_mem, src, src_stride, w, h, border, x0, y0, rows, c, c0); break;
      case 3: median_stage<T, K, 3>(median_mem, src, src_stride, w, h, border, x0, y0, rows, c, c0); break;
      default: median_stage<T, K, 4>(median_mem, src, src_stride, w, h, border, x0, y0, rows, c, c0); break;
    }
    __syncthreads();
    const int x = x0 + CW * lane;
    for (int u = warp; u < channels * (rows / GROUP); u += 4) {
      const int ch = u % channels, y = y0 + u / channels * GROUP;
      if (y >= h) break;
      const uint32_t *base = median_mem + (ch * stage_rows + u / channels * GROUP) * P + CW * lane;
      auto load_row = [&](int i, uint32_t (&v)[CC]) {
        const uint32_t *s = base + i * P;
#pragma unroll
        for (int k = 0; k < CC; k += CW) {
          if constexpr (CW == 4) {
            if (k + 4 <= CC) {
              const uint4 q = *reinterpret_cast<const uint4 *>(s + k);
              v[k] = q.x, v[k + 1] = q.y, v[k + 2] = q.z, v[k + 3] = q.w;
              continue;
            }
          }
          const uint2 q = *reinterpret_cast<const uint2 *>(s + k);
          v[k] = q.x, v[k + 1] = q.y;
        }
      };
      // Per column the K - 1 rows that both output rows read, sorted.
      uint32_t shared[CC][K - 1];
#pragma unroll
      for (int i = 1; i < K; ++i) {
        uint32_t v[CC];
        load_row(i, v);
#pragma unroll
        for (int k = 0; k < CC; ++k) shared[k][i - 1] = v[k];
      }
#pragma unroll
      for (int k = 0; k < CC; ++k) sort_net<PACKED>(shared[k]);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        uint32_t outer[CC], col[CC][K], res[CW];
        load_row(r == 0 ? 0 : K, outer);
#pragma unroll
        for (int k = 0; k < CC; ++k) insert<PACKED, K>(shared[k], outer[k], col[k]);
        static_for<0, CW / 2>([&](auto pc) {
          constexpr int p = 2 * decltype(pc)::value;  // outputs p and p + 1: columns p .. p + K
          uint32_t ml[K][K], mr[K][K];                // their matrices
#pragma unroll
          for (int i = 0; i < K; ++i) {
            uint32_t s[K - 1];
#pragma unroll
            for (int k = 0; k < K - 1; ++k) s[k] = col[p + 1 + k][i];
            sort_net<PACKED>(s);
            insert<PACKED, K>(s, col[p][i], ml[i]);
            insert<PACKED, K>(s, col[p + K][i], mr[i]);
          }
          auto select = [&](const uint32_t (&m)[K][K]) {
            using F = FinalNet<K>;
            uint32_t f[F::wires];
            static_for<0, F::wires>([&](auto ic) {
              constexpr int i = decltype(ic)::value;
              constexpr int row = F::at[i][0], column = F::at[i][1];
              f[i] = m[row][column];
            });
            static_for<0, F::n>([&](auto ic) {
              constexpr int i = decltype(ic)::value;
              constexpr int lo = F::ab[i][0], hi = F::ab[i][1];
              cex<PACKED>(f[lo], f[hi]);
            });
            return f[F::out];
          };
          res[p] = select(ml);
          res[p + 1] = select(mr);
        });
#pragma unroll
        for (int q = 0; q < (PACKED ? 2 : 1); ++q) {
          const int yy = y + r + 2 * q;
          if (yy >= h) continue;
          uint8_t *drow = dst + static_cast<int64_t>(yy) * dst_stride;
          T *d = reinterpret_cast<T *>(drow) + static_cast<int64_t>(x) * c + c0 + ch;
          if constexpr (sizeof(T) == 1 && CW == 4) {
            if (c == 1 && x + 4 <= w && (reinterpret_cast<uintptr_t>(d) & 3) == 0) {
              const uint32_t sel = q ? 0x0062 : 0x0040;  // byte 0 of either half
              const uint32_t flip = static_cast<uint8_t>(Key<T>::from(0)) * 0x01010101u;
              *reinterpret_cast<uint32_t *>(d) =
                  __byte_perm(__byte_perm(res[0], res[1], sel), __byte_perm(res[2], res[3], sel), 0x5410) ^ flip;
              continue;
            }
          }
#pragma unroll
          for (int k = 0; k < CW; ++k)
            if (x + k < w) d[k * c] = Key<T>::from(PACKED ? (q ? res[k] >> 16 : res[k] & 0xFFFFu) : res[k]);
        }
      }
    }
  }
}

constexpr int kHistThreads = 64;

// Pixels per thread: at least K/2, so that the O(K^2) start costs no more per
// pixel than the O(K) steps, and otherwise short, so that a 1080p image still
// gives tens of thousands of threads.
int hist_run(int k) { return std::max(16, (k / 2 + 15) / 16 * 16); }

__global__ void __launch_bounds__(kHistThreads) median_hist_kernel(const uint8_t *src,
                                                                  int64_t src_stride,
                                                                  uint8_t *dst,
                                                                  int64_t dst_stride, int w,
                                                                  int h, int c, int k,
                                                                  int border, int run) {
  __shared__ uint16_t hist[256 * kHistThreads];  // [bin][thread]; counts <= 255 * 255
  launch_dependents();
  grid_dependency_wait();  // the source may be the previous call's output
  const int tid = threadIdx.x;
  const int g = blockIdx.x * kHistThreads + tid;  // (segment, channel) item of a row
  const int ch = g % c, seg = g / c;
  const int x0 = seg * run;
  if (x0 >= w) return;  // no __syncthreads below: threads are independent
  const int x1 = min(w, x0 + run);
  const int r = k / 2;
  const int m = (k * k - 1) / 2;  // rank of the median
  auto value = [&](int yy, int xx) -> int {
    const uint8_t *row = src + static_cast<int64_t>(map_index(yy, h, border)) * src_stride;
    return row[map_index(xx, w, border) * c + ch];
  };
  // Rows loop over the grid's y extent, which the hardware caps at 65535.
  for (int y = blockIdx.y; y < h; y += gridDim.y) {
    for (int b = 0; b < 256; ++b) hist[b * kHistThreads + tid] = 0;
    for (int dy = -r; dy <= r; ++dy)
      for (int dx = -r; dx <= r; ++dx) ++hist[value(y + dy, x0 + dx) * kHistThreads + tid];
    int med = 0, lt = 0;
    while (lt + hist[med * kHistThreads + tid] <= m) lt += hist[(med++) * kHistThreads + tid];
    uint8_t *drow = dst + static_cast<int64_t>(y) * dst_stride;
    drow[x0 * c + ch] = static_cast<uint8_t>(med);
    for (int x = x0 + 1; x < x1; ++x) {
      for (int dy = -r; dy <= r; ++dy) {
        const int out = value(y + dy, x - 1 - r), in = value(y + dy, x + r);
        --hist[out * kHistThreads + tid];
        ++hist[in * kHistThreads + tid];
        lt += (in < med) - (out < med);
      }
      while (lt > m) lt -= hist[(--med) * kHistThreads + tid];
      while (lt + hist[med * kHistThreads + tid] <= m) lt += hist[(med++) * kHistThreads + tid];
      drow[x * c + ch] = static_cast<uint8_t>(med);
    }
  }
}

// Launch under programmatic dependent launch, as the other single calls.
template <typename... P, typename... A>
cudaError_t launch_early(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(static_cast<unsigned>(threads));
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <typename T, int K>
cudaError_t launch_small(const MedianJob &j, cudaStream_t s) {
  constexpr bool PACKED = sizeof(T) <= 2;
  constexpr int tx = 32 * median_width(K), group = median_group(PACKED);
  const int columns = (j.width + tx - 1) / tx;
  auto blocks = [&](int rows) { return static_cast<long>(columns) * ((j.height + rows - 1) / rows); };
  // A block of its own for every channel where blocks of all channels would
  // leave the GPU (three resident per SM) short of a wave, although each then
  // reads every cache line of the image.  All channels in a block against one:
  // 640x480x3 K = 5 / 7 8.3 / 16.7 us against 5.7 / 12.3 us, 1024x768x3 (384 and
  // 768 blocks) 14.2 / 31.9 against 13.2 / 30.1, 1280x720x3 (450 and 900) 14.1 /
  // 32.3 against 14.6 / 33.8.  A block of K = 7 is half as wide, hence twice the
  // count.
  constexpr long kLayerBlocks = 1600 / median_width(K);
  const int layers = blocks(4 * group) < kLayerBlocks ? j.channels : 1;
  // Four warps on 4 groups of rows; fewer groups (all warps still stage) below
  // one and a half such blocks per SM.  640x480x1 (150, 300 or 600 blocks of 16,
  // 8 or 4 rows) K = 5: 16 rows 4.7 us, 8 rows 3.9 us, 4 rows 5.3 us.
  int rows = 4 * group;
  while (rows > group && blocks(rows) * layers < 228) rows /= 2;
  const int row_blocks = (j.height + rows - 1) / rows;
  dim3 grid(static_cast<unsigned>(columns), static_cast<unsigned>(row_blocks < 65535 ? row_blocks : 65535),
            static_cast<unsigned>(layers));
  // At most 38,016 bytes (packed, four channels, K = 5).
  const size_t smem =
      sizeof(uint32_t) * (j.channels / layers) * median_stage_rows(rows, K, PACKED) * median_pitch(K);
  return launch_early(median_small_kernel<T, K>, grid, 128, smem, s, j.src, j.src_stride, j.dst, j.dst_stride,
                      j.width, j.height, j.channels, j.border, rows);
}

template <typename T>
cudaError_t launch3(const MedianJob &j, cudaStream_t s) {
  const int row_blocks = (j.height + 3) / 4;
  dim3 grid(static_cast<unsigned>((j.width * j.channels + 127) / 128),
            static_cast<unsigned>(row_blocks < 65535 ? row_blocks : 65535));
  return launch_early(median3_kernel<T>, grid, 128, 0, s, j.src, j.src_stride, j.dst, j.dst_stride, j.width, j.height,
                      j.channels, j.border);
}

template <typename T>
cudaError_t launch_typed(const MedianJob &j, cudaStream_t s) {
  switch (j.ksize) {
    case 3: return launch3<T>(j, s);
    case 5: return launch_small<T, 5>(j, s);
    case 7: return launch_small<T, 7>(j, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_median(const MedianJob &j, cudaStream_t s) {
  if (j.ksize > 7) {
    if (j.elem != MEDIAN_U8) return cudaErrorInvalidValue;
    const int run = hist_run(j.ksize);
    const int items = j.channels * ((j.width + run - 1) / run);
    dim3 grid(static_cast<unsigned>((items + kHistThreads - 1) / kHistThreads),
              static_cast<unsigned>(j.height < 65535 ? j.height : 65535));
    return launch_early(median_hist_kernel, grid, kHistThreads, 0, s, j.src, j.src_stride, j.dst, j.dst_stride,
                        j.width, j.height, j.channels, j.ksize, j.border, run);
  }
  switch (j.elem) {
    case MEDIAN_S8: return launch_typed<int8_t>(j, s);
    case MEDIAN_U8: return launch_typed<uint8_t>(j, s);
    case MEDIAN_U16: return launch_typed<uint16_t>(j, s);
    case MEDIAN_S16: return launch_typed<int16_t>(j, s);
    case MEDIAN_U32: return launch_typed<uint32_t>(j, s);
    case MEDIAN_S32: return launch_typed<int32_t>(j, s);
    case MEDIAN_F32: return launch_typed<float>(j, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace kcv
