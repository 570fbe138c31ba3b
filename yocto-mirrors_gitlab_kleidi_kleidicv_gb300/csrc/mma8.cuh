// u8 separable stencils on the tensor cores (sm_103a): gaussian_blur_u8 with
// generated weights of any size (3..255) and with the binomial kernels of
// sizes 3 and 5, and the u8 separable filter.
//
// Both passes are products with a banded (Toeplitz) weight matrix, on
// mma.sync.m16n8k16 (f16 operands, f32 accumulators):
//
//   V[y][x] = sum_k Wy[y][k] S[k][x]     per mma 8 rows x 16 columns of V
//   D[y][x] = sum_k V[y][k] Wx[k][x]     per mma 16 rows x 8 bytes of D
//
// The vertical band of 8 rows covers 8 + K - 1 source rows, the horizontal
// one of 8 bytes 8 + (K - 1) C bytes of V (tap distance C bytes, the other
// entries zero).
//
// Exactness.  A byte v in the low half of a 16-bit word is the f16 subnormal
// v * 2^-24, so bytes become operands by a mask, without a conversion.
// Weights (integers 0..255) are exact in f16, every product is an integer
// multiple of 2^-24 and every sum of a pass stays below 2^19 multiples, so
// the f32 accumulator, which starts at 0.5 + 128 * 2^-24 (0.5 for the
// separable filter), holds each partial sum exactly: its bits are
// 0x3F000000 + (128 + sum), and the reference's (128 + sum) >> 8 is bits 8..15
// of the register (gaussian_blur_fixed_neon.cpp:501-526 and the horizontal
// pass after it; gaussian_blur_arbitrary_neon.cpp:193-383 for the larger
// sizes, whose saturating and wrapping elements are told apart below).  The
// saturating u8 filter (separable_filter_2d_neon.cpp:38-136, taps >= 0) takes
// min(sum, 255) of both passes.
//
// Why tensor cores for a stencil: a tap costs an element one half-rate
// integer instruction per pass and lane pair, so the kernels that multiply
// in integer lanes were bound by issue from about 9 taps on; an mma takes 8
// cycles of a sub-core for 2048 multiply-adds, of which a K-tap band uses
// K / 16 at K <= 9, K / 32 at K <= 25.  mma.sync rather than tcgen05: a tile
// of 8 rows needs a band 8 + K - 1 deep where the 128 rows of a tcgen05 tile
// need 128 + K - 1, and no operand has to be written to shared memory in a
// descriptor's layout.
//
// A CTA computes tiles of 16 MT rows x W = 256 bytes:
//   stage   source rows (border-mapped) and columns [x0 - hp, x0 + W + rc) in one
//           of two shared-memory buffers, behind the passes of the tile before:
//           16-byte cp.async where base and stride allow, else two aligned
//           16-byte loads and a funnel shift; columns outside the row are
//           written afterwards, one byte per thread, from the staged row;
//   pass 1  a warp takes blocks of 16 columns; ldmatrix.trans gives rows
//           (2t, 2t + 1) of byte pair g in one register, whose even and odd bytes
//           are the A operands of the block's even and odd columns, and 8 source
//           rows serve every group of 8 destination rows that reads them;
//           results go to shared memory as bytes;
//   pass 2  a warp takes 16 rows x RUN bytes; ldmatrix gives four bytes of a row
//           per register, whose even and odd bytes are A operands (the weight
//           matrix is permuted to match); the window of blocks slides through
//           registers, and the results leave through a per-warp staging area
//           as 16-byte (or aligned 4-byte) stores.
// Row pitches are odd multiples of 16 bytes: the 8 rows of an ldmatrix phase
// lie in distinct bank groups.  Nine warps: the 18 column blocks of a tile
// are two per warp (eight warps took three turns for them); eight units of
// pass 2.
//
// Measured (GB300, back to back; before: the tiled and the two-pass kernel):
// 3840x2160x1 31 taps 132 -> 10.7 us, 255 taps 873 -> 77 us; 3840x2160x3 15
// taps 66 -> 22.9 us, 1917x1079x3 (unaligned rows) 48.3 -> 13.9 us;
// 3840x2160x4 21 taps 134 -> 43.1 us; 1920x1080x1 7 taps 9.3 -> 4.1 us.
// No pipe is full: 3840x2160x1 at 7 / 31 / 101 / 255 taps uses 44 / 42 / 34 /
// 33 % of the issue slots and 19 / 34 / 37 / 43 % of the tensor pipe's cycles,
// with 25 % of the warps resident, and 14 % (shared memory for one CTA) at 101
// and 255 taps.  At 31 taps a warp takes 9.7 cycles per instruction: 1.9 in
// fixed waits, 1.7 for the tensor pipe, 1.6 at the CTA's barriers, 0.7 for shared
// memory, 0.65 for instructions, 0.4 for global loads; with unaligned rows
// (1917x1079x3, 15 taps) 2.1 of 9.4 are for global loads and 1.0 at barriers.  Three CTAs of 72
// registers per thread spill: 1920x1080x1 7 taps 4.9 us.  7 taps are 99 warp
// instructions per 16 x 16 bytes; unaligned rows take 1.7 times as many.
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

#include "kcv_job.h"
#include "ptx.cuh"
#include "sepfused.cuh"

namespace kcv {

constexpr int kMma8Warps = 9;
constexpr int kMma8Threads = 32 * kMma8Warps;
// Destination bytes of a warp's unit of pass 2 (a tile is eight units) and
// its staging area of 16 rows.
__host__ __device__ constexpr int mma8_run(int mt, int w) { return mt * w / 8; }
__host__ __device__ constexpr int mma8_out_pitch(int run) { return run + 16; }
__host__ __device__ constexpr int mma8_out_bytes(int run) { return kMma8Warps * 16 * mma8_out_pitch(run); }

// How sums become bytes: bits 8..15 (weights sum to at most 256); the same
// with the saturation and the right-border lanes of the arbitrary-size path;
// min(sum, 255); the binomial kernels of sizes 3 and 5, whose vertical sums
// are not rounded (gaussian_blur_fixed_neon.cpp:27-153).  Those sums (at most
// 1020 or 4080) are formed times 64 or 16, below 2^16, so that their high and
// low bytes are byte results like the others; pass 2 multiplies the planes of
// high and low bytes with the weights times 64 (16) and divided by 4 (16), all
// exact, which gives 16 (1) times the binomial sum.
enum Mma8Epi { kEpiRound = 0, kEpiArbitrary = 1, kEpiSat8 = 2, kEpiBinomial = 3 };

__host__ __device__ constexpr int mma8_round16(int v) { return (v + 15) / 16 * 16; }
// Row pitch: an odd multiple of 16 bytes.
__host__ __device__ constexpr int mma8_pitch(int cols) { return (mma8_round16(cols) / 16 | 1) * 16; }

// Shared-memory geometry of an instantiation: known at compile time (so that
// every offset is an immediate) where both step counts are, else the job's.
template <int NK, int NB, int MT, int W>
struct Mma8Geo {
  static constexpr bool kFixed = NK > 0 && NB > 0;
  // NB steps hold a halo of at most 8 (NB - 1) bytes on either side.
  static constexpr int kHalo = mma8_round16(8 * (NB - 1));
  static constexpr int kRawRows = 8 * (2 * MT + 2 * NK - 1);
  static constexpr int kRawCols = W + 2 * kHalo;
  static constexpr int kRawPitch = mma8_pitch(kRawCols);
  static constexpr int kVCols = W + 16 * (NB - 1);
  static constexpr int kVPitch = mma8_pitch(kVCols);
  __device__ static int raw_pitch(const Mma8Job &j) { return kFixed ? kRawPitch : j.raw_pitch; }
  __device__ static int raw_cols(const Mma8Job &j) { return kFixed ? kRawCols : j.raw_cols; }
  __device__ static int raw_rows(const Mma8Job &j) { return kFixed ? kRawRows : j.raw_rows; }
  __device__ static int v_pitch(const Mma8Job &j) { return kFixed ? kVPitch : j.v_pitch; }
  __device__ static int v_cols(const Mma8Job &j) { return kFixed ? kVCols : j.v_cols; }
};

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// d = a * b + c.
__device__ __forceinline__ void mma_f16_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1,
                                              const float (&c)[4]) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c[0]), "f"(c[1]), "f"(c[2]), "f"(c[3]));
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm_x1_trans(uint32_t &r0, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x1.trans.shared.b16 {%0}, [%1];" : "=r"(r0) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x2_trans(uint32_t &r0, uint32_t &r1, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(r0), "=r"(r1)
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void sts16(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.u16 [%0], %1;" ::"r"(addr), "h"(static_cast<uint16_t>(v)) : "memory");
}
// Even / odd bytes of a word as a pair of f16 subnormals.
__device__ __forceinline__ uint32_t even_bytes(uint32_t w) { return w & 0x00FF00FFu; }
__device__ __forceinline__ uint32_t odd_bytes(uint32_t w) { return __byte_perm(w, 0u, 0x4341); }

// The accumulators' first value.  Four opaque registers: as known constants
// they are copied into place before every first mma (four moves each, a
// sixth of the kernel's instructions).
template <bool ROUND>
__device__ __forceinline__ void mma8_init(float (&c)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) asm volatile("mov.b32 %0, %1;" : "=f"(c[i]) : "n"(ROUND ? 0x3F000080 : 0x3F000000));
}
// The result bytes of two sums in the low half of a word.
template <int EPI>
__device__ __forceinline__ uint32_t pack_pair(uint32_t a, uint32_t b) {
  return __byte_perm(a, b, EPI == kEpiSat8 ? 0x0040u : 0x0051u);
}
template <int EPI>
__device__ __forceinline__ uint32_t finish_sum(float acc, bool saturate) {
  const uint32_t bits = __float_as_uint(acc);
  if constexpr (EPI == kEpiSat8) return min(bits, 0x3F0000FFu);
  else if constexpr (EPI == kEpiArbitrary) return saturate ? min(bits, 0x3F00FFFFu) : bits;
  else return bits;
}

__device__ __forceinline__ void cp_async16_z(uint32_t dst, const void *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// The weight operands in fragment order: wa[step][lane] = the two B words of
// the vertical step, wb[step][lane] = the B words of both accumulators of the
// horizontal step.  They are read from the taps spread over source rows and
// over source bytes (zero between the bytes of a channel and around).
constexpr int kTapPad = 32;
constexpr int kTapsY = kTapPad + 255 + 33;           // index kTapPad + row distance
constexpr int kTapsX = kTapPad + 4 * 254 + 1 + 47;   // index kTapPad + byte distance
struct Mma8Taps {
  uint8_t y[kTapsY], x[kTapsX];
};

// Integers 0..1023 as f16: 1024 + v placed by its bits, minus 1024 (exact).
__device__ __forceinline__ uint32_t half_pair(uint32_t lo, uint32_t hi) {
  const uint32_t biased = 0x64006400u | lo | hi << 16, bias = 0x64006400u;
  const __half2 h = __hsub2(*reinterpret_cast<const __half2 *>(&biased), *reinterpret_cast<const __half2 *>(&bias));
  return *reinterpret_cast<const uint32_t *>(&h);
}
__device__ __forceinline__ void clear_taps(Mma8Taps &taps) {
  for (int i = threadIdx.x; i < static_cast<int>(sizeof(taps) / 4); i += kMma8Threads)
    reinterpret_cast<uint32_t *>(&taps)[i] = 0u;
}
__device__ __forceinline__ void spread_taps(const Mma8Job &j, Mma8Taps &taps) {
  for (int i = threadIdx.x; i < j.ksize; i += kMma8Threads) {
    taps.y[kTapPad + i] = j.ty[i];
    taps.x[kTapPad + i * j.c] = j.tx[i];
  }
}
template <int EPI>
__device__ __forceinline__ void build_weights(const Mma8Job &j, const Mma8Taps &taps, uint32_t *wa, uint32_t *wb) {
  const int na = j.nk * 64, n = na + j.nb * 128;
  // Binomial: the vertical weights and those of the high plane times `up`, the
  // low plane's (behind them) times `down`.
  const uint32_t up = EPI == kEpiBinomial ? (j.ksize == 3 ? 64u : 16u) : 1u;
  const __half2 down = __float2half2_rn(j.ksize == 3 ? 0.25f : 0.0625f);
  for (int i = threadIdx.x; i < n; i += kMma8Threads) {
    if (i < na) {
      // B[k][n]: destination row n = g, source rows k = 2t, 2t + 1 (+ 8 in word 1).
      const int l = (i >> 1) & 31, g = l >> 2, t = l & 3;
      const int z = min(16 * (i >> 6) + 2 * t + (i & 1) * 8 - g, 2 * j.r + 1);
      wa[i] = half_pair(up * taps.y[kTapPad + z], up * taps.y[kTapPad + z + 1]);
    } else {
      // B[k][n] of accumulator p: destination byte n + 8p, k = bytes 4t + e and
      // 4t + e + 2 of the step's block (e = word & 1).
      const int w = i - na, l = (w >> 2) & 31, g = l >> 2, t = l & 3;
      const int z = min(16 * (w >> 7) + 4 * t + (w & 1) - j.vo - (g + 4 * (w & 2)) + j.rc, 2 * j.rc + 1);
      const uint32_t lo = taps.x[kTapPad + z], hi = taps.x[kTapPad + z + 2];
      wb[w] = half_pair(up * lo, up * hi);
      if constexpr (EPI == kEpiBinomial) {
        const uint32_t h = half_pair(lo, hi);
        const __half2 q = __hmul2(*reinterpret_cast<const __half2 *>(&h), down);
        wb[j.nb * 128 + w] = *reinterpret_cast<const uint32_t *>(&q);
      }
    }
  }
}

// Source byte offset of row byte x (outside [0, wc)) under the border, or -1
// for the border value.
__device__ __forceinline__ int border_byte(const Mma8Job &j, int x) {
  const int bias = j.c * 256;  // x >= -rc > -bias
  const int col = (x + bias) / j.c - 256;
  const int m = map_index(col, j.w, j.border);
  return m < 0 ? -1 : m * j.c + (x - col * j.c);
}

struct Mma8Smem {
  uint32_t *wa, *wb;
  uint8_t *raw, *v;  // raw: the buffer of the current step
};

// Stages `rows` source rows from y0 on (mapped to the image) of the columns
// [xb, xb + 16 np).  A thread keeps its 16-byte piece of the row (piece p0 + p,
// np <= 97) and steps down the rows.  NP: np where it is known, else 0.
template <int NP, bool ALIGNED>
__device__ __forceinline__ void stage_pieces(const Mma8Job &j, uint8_t *raw, int pitch, int y0, int rows, int xb, int p0,
                                             int np_) {
  const int np = NP > 0 ? NP : np_;
  const uint32_t bv = (static_cast<uint32_t>(j.border_value) & 0xFFu) * 0x01010101u;
  const int step = kMma8Threads / np;
  const int row0 = static_cast<int>(threadIdx.x) / np;
  if (row0 >= step) return;
  const int p = p0 + static_cast<int>(threadIdx.x) - row0 * np;
  const uint8_t *const base = j.src + xb + 16 * p;
  const int avail = j.wc - xb - 16 * p;  // bytes of the row from there on
  int off = row0 * pitch + 16 * p;
  if constexpr (ALIGNED) {
    const int n = min(16, avail);
    if (y0 >= 0 && y0 + rows <= j.h) {
      // Consecutive rows of the image.
      const uint8_t *g = base + static_cast<int64_t>(y0 + row0) * j.src_stride;
      const int64_t gstep = static_cast<int64_t>(step) * j.src_stride;
      uint32_t a = smem_addr(raw) + off;
      for (int row = row0; row < rows; row += step, g += gstep, a += step * pitch) cp_async16_z(a, g, n);
      return;
    }
    for (int row = row0; row < rows; row += step, off += step * pitch) {
      const int y = map_index(y0 + row, j.h, j.border);
      if (y < 0) *reinterpret_cast<uint4 *>(raw + off) = make_uint4(bv, bv, bv, bv);
      else cp_async16_z(smem_addr(raw) + off, base + static_cast<int64_t>(y) * j.src_stride, n);
    }
  } else {
    // The two aligned blocks around the piece, where they lie in the image
    // (bytes of the neighbouring rows are replaced or never read), loaded for
    // two rows before the first is shifted and stored.  The 512-image batch with
    // 1 / 2 / 3 / 5 rows: 998 / 942 / 988 / 1204 us; the batch kernels spill up
    // to 32 / 84 / 224 bytes at 2 / 3 / 5.
    const uint8_t *const end = j.src + static_cast<int64_t>(j.h - 1) * j.src_stride + j.wc;
    constexpr int kAhead = 2;
    for (int row = row0; row < rows; row += kAhead * step, off += kAhead * step * pitch) {
      uint4 u[kAhead], v[kAhead];
      int sh[kAhead];  // -1: nothing loaded
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        sh[k] = -1;
        const int y = row + k * step < rows ? map_index(y0 + row + k * step, j.h, j.border) : -1;
        const uint8_t *g = base + static_cast<int64_t>(y) * j.src_stride;
        const int m = static_cast<int>(reinterpret_cast<uintptr_t>(g) & 15);
        if (y >= 0 && g - m >= j.src && g - m + 32 <= end) {
          u[k] = ld_src_v4(g - m);
          v[k] = ld_src_v4(g - m + 16);
          sh[k] = m;
        }
      }
#pragma unroll
      for (int k = 0; k < kAhead; ++k) {
        uint8_t *d = raw + off + k * step * pitch;
        if (sh[k] >= 0) {
          *reinterpret_cast<uint4 *>(d) = shift_blocks(u[k], v[k], sh[k]);
        } else if (row + k * step < rows) {
          const int y = map_index(y0 + row + k * step, j.h, j.border);
          if (y < 0) {
            *reinterpret_cast<uint4 *>(d) = make_uint4(bv, bv, bv, bv);
          } else {
            const uint8_t *g = base + static_cast<int64_t>(y) * j.src_stride;
            for (int i = 0; i < min(16, avail); ++i) d[i] = ld_src(g + i);
          }
        }
      }
    }
  }
}
template <typename G>
__device__ __forceinline__ void stage_columns(const Mma8Job &j, uint8_t *raw, int y0, int rows, int xb, int ncols,
                                              int xe) {
  // Pieces of 16 bytes lying at least partly inside the row.
  const int p0 = xb < 0 ? -xb >> 4 : 0;
  const int np = ((min(min(xb + ncols, xe), j.wc) - xb + 15) >> 4) - p0;
  const int pitch = G::raw_pitch(j);
  if (((reinterpret_cast<uintptr_t>(j.src) | static_cast<uintptr_t>(j.src_stride)) & 15) == 0) {
    if (G::kFixed && np == G::kRawCols / 16)  // an inner tile
      stage_pieces<G::kFixed ? G::kRawCols / 16 : 1, true>(j, raw, pitch, y0, rows, xb, p0, np);
    else if (np > 0)
      stage_pieces<0, true>(j, raw, pitch, y0, rows, xb, p0, np);
  } else if (np > 0) {
    stage_pieces<0, false>(j, raw, pitch, y0, rows, xb, p0, np);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}

// Columns outside the row: every thread takes one column (its mapped source
// column computed once) and walks down the rows.  Call after the staged
// pieces are visible to the CTA.
__device__ __forceinline__ bool has_border_columns(const Mma8Job &j, int xb, int ncols, int xe) {
  return xb < 0 || min(xb + ncols, xe) > j.wc;
}
__device__ __forceinline__ void fill_border_columns(const Mma8Job &j, uint8_t *raw, int pitch, int y0, int rows, int xb,
                                                    int ncols, int xe) {
  const int l0 = max(xb, -j.rc), l1 = min(xb + ncols, 0);
  const int r0 = max(xb, j.wc), r1 = min(xb + ncols, xe);
  const int nl = max(0, l1 - l0), nr = max(0, r1 - r0), n = nl + nr;
  const uint8_t bv = static_cast<uint8_t>(j.border_value);
  for (int base = 0; base < n; base += kMma8Threads) {
    const int nn = min(n - base, kMma8Threads);
    const int step = kMma8Threads / nn;
    const int row0 = static_cast<int>(threadIdx.x) / nn, q = static_cast<int>(threadIdx.x) - row0 * nn + base;
    if (row0 >= step) continue;
    const int x = q < nl ? l0 + q : r0 + (q - nl);
    const int from = border_byte(j, x);
    const bool local = from >= max(xb, 0) && from < min(min(xb + ncols, xe), j.wc);
    for (int row = row0; row < rows; row += step) {
      uint8_t v = bv;
      if (local) {  // a CONSTANT row was staged as the border value
        v = raw[row * pitch + from - xb];
      } else if (from >= 0) {
        const int y = map_index(y0 + row, j.h, j.border);
        if (y >= 0) v = ld_src(j.src + static_cast<int64_t>(y) * j.src_stride + from);
      }
      raw[row * pitch + x - xb] = v;
    }
  }
}

// Pass 1 over the staged columns [xb, xb + ncols) of the tile at x0: per
// block of 16 columns and group of 8 destination rows, D[column][row] with
// the source as the A operand (even columns in its rows 0..7, odd ones in
// 8..15).  Group i reads the 8-row matrices i .. i + 2 NK - 1.
template <int NK, int NB, int MT, int W, int EPI>
__device__ __forceinline__ void vertical_pass(const Mma8Job &j, const Mma8Smem &s, int x0, int xb, int ncols) {
  using G = Mma8Geo<NK, NB, MT, W>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  float init[4];
  mma8_init<EPI == kEpiRound || EPI == kEpiArbitrary>(init);
  const uint2 *wa = reinterpret_cast<const uint2 *>(s.wa);
  const int rp = G::raw_pitch(j), vp = G::v_pitch(j);
  const uint32_t raw = smem_addr(s.raw) + lane * rp;  // the lane's row of ldmatrix loads
  const int v0 = xb - x0 + j.vo + 2 * g;              // the lane's V columns of block 0: v0, v0 + 1
  const uint32_t vbase = smem_addr(s.v) + 2 * t * vp + v0;  // rows 2t, 2t + 1 of a group
  const bool sat = EPI == kEpiArbitrary && j.saturate != 0;
  auto store = [&](const float (&acc)[4], int group, uint32_t v) {
    v += 8 * group * vp;
    if constexpr (EPI == kEpiBinomial) {
      const uint32_t c[4] = {__float_as_uint(acc[0]), __float_as_uint(acc[1]), __float_as_uint(acc[2]),
                             __float_as_uint(acc[3])};
      sts16(v, __byte_perm(c[0], c[2], 0x0051));
      sts16(v + vp, __byte_perm(c[1], c[3], 0x0051));
      sts16(v + 16 * MT * vp, __byte_perm(c[0], c[2], 0x0040));
      sts16(v + 16 * MT * vp + vp, __byte_perm(c[1], c[3], 0x0040));
      return;
    }
    sts16(v, pack_pair<EPI>(finish_sum<EPI>(acc[0], sat), finish_sum<EPI>(acc[2], sat)));
    sts16(v + vp, pack_pair<EPI>(finish_sum<EPI>(acc[1], sat), finish_sum<EPI>(acc[3], sat)));
  };
  if constexpr (NK > 0) {
    uint2 w[NK];
#pragma unroll
    for (int d = 0; d < NK; ++d) w[d] = wa[d * 32 + lane];
    constexpr int kMats = 2 * MT + 2 * NK - 1;
    for (int q = warp; q < ncols / 16; q += kMma8Warps) {
      const bool inside = v0 + 16 * q >= 0 && v0 + 16 * q < G::v_cols(j);
      const uint32_t vq = vbase + 16 * q, rq = raw + 16 * q;
      float accs[2][4];
      uint32_t e[kMats], o[kMats];  // few are live at a time
      static_for<0, kMats>([&](auto mc) {
        constexpr int m = decltype(mc)::value;
        if constexpr (m % 4 == 0) {
          uint32_t r[4];
          const uint32_t a = rq + 8 * m * rp;
          constexpr int n = kMats - m < 4 ? kMats - m : 4;
          if constexpr (n == 4) ldsm_x4_trans(r, a);
          if constexpr (n == 2 || n == 3) ldsm_x2_trans(r[0], r[1], a);
          if constexpr (n == 3) ldsm_x1_trans(r[2], a + 16 * rp);
          if constexpr (n == 1) ldsm_x1_trans(r[0], a);
#pragma unroll
          for (int k = 0; k < n; ++k) e[m + k] = even_bytes(r[k]), o[m + k] = odd_bytes(r[k]);
        }
        // Group m - 2 NK + 1 has its last matrix.
        if constexpr (m >= 2 * NK - 1) {
          constexpr int i = m - 2 * NK + 1;
          // A group's results are stored behind the next group's products.
          float(&acc)[4] = accs[i % 2];
          static_for<0, NK>([&](auto dc) {
            constexpr int d = decltype(dc)::value;
            const uint32_t a[4] = {e[i + 2 * d], o[i + 2 * d], e[i + 2 * d + 1], o[i + 2 * d + 1]};
            if constexpr (d == 0) mma_f16_first(acc, a, w[d].x, w[d].y, init);
            else mma_f16(acc, a, w[d].x, w[d].y);
          });
          if constexpr (i > 0)
            if (inside) store(accs[(i + 1) % 2], i - 1, vq);
        }
      });
      if (inside) store(accs[(2 * MT - 1) % 2], 2 * MT - 1, vq);
    }
  } else {
    static_assert(MT == 4, "the weight slots rotate by four");
    for (int q = warp; q < ncols / 16; q += kMma8Warps) {
      float acc[8][4];
      uint2 w[4];  // w[d % 4]: vertical step d, zero outside the band
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[i][k] = init[k];
#pragma unroll
      for (int d = 0; d < 4; ++d) w[d] = make_uint2(0u, 0u);
      uint32_t r0;
      ldsm_x1_trans(r0, raw + 16 * q);
      uint32_t e0 = even_bytes(r0), o0 = odd_bytes(r0);
      const int steps = j.nk + 3;
      for (int db = 0; db < steps; db += 4) {
        static_for<0, 4>([&](auto dc) {
          constexpr int dd = decltype(dc)::value;
          const int d = db + dd;
          if (d >= steps) return;
          w[dd] = d < j.nk ? wa[d * 32 + lane] : make_uint2(0u, 0u);
          // Matrices 2d (carried over), 2d + 1 and 2d + 2.
          uint32_t r1, r2;
          ldsm_x2_trans(r1, r2, raw + (16 * d + 8) * rp + 16 * q);
          const uint32_t a[4] = {e0, o0, even_bytes(r1), odd_bytes(r1)};
          e0 = even_bytes(r2), o0 = odd_bytes(r2);
          const uint32_t b[4] = {a[2], a[3], e0, o0};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            mma_f16(acc[2 * i], a, w[(dd - i + 4) % 4].x, w[(dd - i + 4) % 4].y);
            mma_f16(acc[2 * i + 1], b, w[(dd - i + 4) % 4].x, w[(dd - i + 4) % 4].y);
          }
        });
      }
      if (v0 + 16 * q >= 0 && v0 + 16 * q < G::v_cols(j)) {
#pragma unroll
        for (int i = 0; i < 8; ++i) store(acc[i], i, vbase + 16 * q);
      }
    }
  }
}

// The arbitrary-size path's right-border vectors read, for taps wholly past
// the row end, another channel of the last pixel in their last lanes
// (border_generic_neon.h:80-98, gaussian_blur_arbitrary_neon.cpp:346-377):
// the vector starting at xv (8 elements, the first at wc - arb_border_len)
// has q = (xv - wc) mod c, and its lanes 8 - q .. 7 read channel lane + c - 8
// for every tap distance d with xv + c d >= wc.  Returns the sum's correction
// for destination byte x of the V row `vrow` (column 0 at byte x0 - vo).
static __device__ __noinline__ uint32_t right_lane_correction(const Mma8Job &j, const uint8_t *vrow, int x0, int x) {
  const int start = j.wc - j.arb_border_len;
  if (x < start) return 0u;
  const int xv = start + (x - start) / 8 * 8, lane = x - xv;
  const int d0 = (j.wc - xv + j.c - 1) / j.c;
  const int q = xv + j.c * d0 - j.wc;
  if (q == 0 || lane < 8 - q) return 0u;
  const uint8_t *v = vrow + j.vo - x0;  // v[byte of the row]
  const uint32_t last = v[j.wc - j.c + lane + j.c - 8];
  uint32_t corr = 0;
  for (int d = d0; d <= j.r; ++d) corr += j.tx[j.r + d] * (last - v[x + j.c * d]);
  return corr;
}

// Staged rows (`rows` of 16) x n bytes (n <= 16 kPieces) to the destination
// rows from `d` on, whole or in part and whatever their alignment.
template <int kPieces>
__device__ __forceinline__ void store_ragged(const Mma8Job &j, const uint8_t *stg, uint8_t *d, int rows, int n, int lane,
                                             bool aligned) {
  constexpr int kPitch = 16 * kPieces + 16;
  if (aligned) {
    constexpr int kRows = 32 / kPieces;  // rows at a time
    const int p = lane % kPieces;
#pragma unroll 1
    for (int row = lane / kPieces; row < rows; row += kRows) {
      uint8_t *dd = d + static_cast<int64_t>(row) * j.dst_stride + 16 * p;
      const uint8_t *sp = stg + row * kPitch + 16 * p;
      if (16 * p + 16 <= n) {
        *reinterpret_cast<uint4 *>(dd) = *reinterpret_cast<const uint4 *>(sp);
      } else {
        for (int i = 0; i < n - 16 * p; ++i) dd[i] = sp[i];
      }
    }
    return;
  }
  // Aligned 16-byte blocks of the destination, each from the two staged blocks
  // around it; then the bytes before the first and after the last of them, one
  // lane per row and end, as pieces of 1, 2, 4 and 8 bytes.
  constexpr int kRows = 32 / kPieces;
  const int p = lane % kPieces;
#pragma unroll 2
  for (int row = lane / kPieces; row < rows; row += kRows) {
    uint8_t *dd = d + static_cast<int64_t>(row) * j.dst_stride;
    const int head = static_cast<int>(-reinterpret_cast<uintptr_t>(dd) & 15);  // bytes before the first block
    if (head + 16 * p + 16 <= n) {
      const uint8_t *sp = stg + row * kPitch + 16 * p;
      const uint4 u = *reinterpret_cast<const uint4 *>(sp), v = *reinterpret_cast<const uint4 *>(sp + 16);
      *reinterpret_cast<uint4 *>(dd + head + 16 * p) = shift_blocks(u, v, head);
    }
  }
  const int row = lane >> 1;
  if (row >= rows) return;
  uint8_t *dd = d + static_cast<int64_t>(row) * j.dst_stride;
  const uint8_t *sp = stg + row * kPitch;
  const uint32_t *sw = reinterpret_cast<const uint32_t *>(sp);
  const int head = static_cast<int>(-reinterpret_cast<uintptr_t>(dd) & 15);
  if (head > n) {  // no whole block: a narrow last run
    if ((lane & 1) == 0)
      for (int i = 0; i < n; ++i) dd[i] = sp[i];
    return;
  }
  const bool tail = (lane & 1) != 0;
  const int from = tail ? head + (n - head) / 16 * 16 : 0;  // first byte of the end
  const int c = tail ? n - from : head;                     // and its bytes
  auto word = [&](int o) { return __funnelshift_r(sw[o >> 2], sw[(o >> 2) + 1], 8 * (o & 3)); };
  if (c & 8) {
    const int o = from + (tail ? 0 : c & 7);
    *reinterpret_cast<uint2 *>(dd + o) = make_uint2(word(o), word(o + 4));
  }
  if (c & 4) {
    const int o = from + (tail ? c & 8 : c & 3);
    *reinterpret_cast<uint32_t *>(dd + o) = word(o);
  }
  if (c & 2) {
    const int o = from + (tail ? c & 12 : c & 1);
    *reinterpret_cast<uint16_t *>(dd + o) = static_cast<uint16_t>(word(o));
  }
  if (c & 1) {
    const int o = from + (tail ? c & 14 : 0);
    dd[o] = sp[o];
  }
}

template <int NK, int NB, int NA, int MT, int W, int EPI>
__device__ __forceinline__ void horizontal_pass(const Mma8Job &j, const Mma8Smem &s, int x0, int y0, int we, int rows) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t = lane & 3;
  float init[4];
  mma8_init<EPI != kEpiSat8>(init);
  const uint4 *wb = reinterpret_cast<const uint4 *>(s.wb);
  const int vp = Mma8Geo<NK, NB, MT, W>::v_pitch(j);
  constexpr int RUN = mma8_run(MT, W), kBlocks = RUN / 16, kPitch = mma8_out_pitch(RUN);
  uint8_t *const stg = s.raw + warp * 16 * kPitch;  // the staged source is dead
  const uint32_t stp = smem_addr(stg) + g * kPitch + 2 * t;
  if (warp < 8) {
    const int m = warp % MT, run = warp / MT;
    const int mrows = min(16, rows - 16 * m);
    const int n = min(RUN, we - RUN * run);
    if (mrows <= 0 || n <= 0) return;
    const int nblk = (n + 15) / 16;
    // ldmatrix rows: lanes 0..15 the 16 rows of a block, 16..31 of the next one.
    const uint32_t va = smem_addr(s.v) + (16 * m + (lane & 15)) * vp + RUN * run + (lane >> 4) * 16;
    auto finish = [&](float (&acc)[2][4], int b) {
      uint32_t w[2][4];
#pragma unroll
      for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int i = 0; i < 4; ++i) w[p][i] = __float_as_uint(acc[p][i]);
      if constexpr (EPI == kEpiArbitrary) {
        const int x = x0 + RUN * run + 16 * b + 2 * t;  // accumulator p: bytes x + 8p, x + 8p + 1
        const bool right = j.quirk && x + 16 > j.wc - j.arb_border_len;
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int xe = x + 8 * p + (i & 1);
            if (right && xe < j.wc)
              w[p][i] += right_lane_correction(j, s.v + (16 * m + g + 8 * (i >> 1)) * vp, x0, xe);
            w[p][i] = finish_sum<EPI>(__uint_as_float(w[p][i]), xe >= j.h_sat_from && xe < j.h_sat_to);
          }
      } else {
#pragma unroll
        for (int p = 0; p < 2; ++p)
#pragma unroll
          for (int i = 0; i < 4; ++i) w[p][i] = finish_sum<EPI>(acc[p][i], false);
      }
#pragma unroll
      for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh)
          sts16(stp + 8 * hh * kPitch + 16 * b + 8 * p, pack_pair<EPI>(w[p][2 * hh], w[p][2 * hh + 1]));
    };
    if constexpr (NB > 0) {
      uint32_t wr[NB][4];
#pragma unroll
      for (int k = 0; k < NB; ++k) {
        const uint4 w = wb[k * 32 + lane];
        wr[k][0] = w.x, wr[k][1] = w.y, wr[k][2] = w.z, wr[k][3] = w.w;
      }
      // win[k % (NB + 1)]: the A operand of block k, loaded in pairs; of the
      // plane of low bytes in wlo with its weights wrl.
      constexpr bool kPlanes = EPI == kEpiBinomial;
      uint32_t win[NB + 1][4], wlo[kPlanes ? NB + 1 : 1][4], wrl[kPlanes ? NB : 1][4];
      if constexpr (kPlanes) {
#pragma unroll
        for (int k = 0; k < NB; ++k) {
          const uint4 w = wb[(NB + k) * 32 + lane];
          wrl[k][0] = w.x, wrl[k][1] = w.y, wrl[k][2] = w.z, wrl[k][3] = w.w;
        }
      }
      float accs[2][2][4];
      auto load_pair = [&](auto kc) {
        constexpr int k = decltype(kc)::value;
        auto load = [&](uint32_t addr, uint32_t(&w0)[4], uint32_t(&w1)[4]) {
          uint32_t r[4];
          ldsm_x4(r, addr);
          w0[0] = even_bytes(r[0]), w0[1] = even_bytes(r[1]), w0[2] = odd_bytes(r[0]), w0[3] = odd_bytes(r[1]);
          w1[0] = even_bytes(r[2]), w1[1] = even_bytes(r[3]), w1[2] = odd_bytes(r[2]), w1[3] = odd_bytes(r[3]);
        };
        load(va + 16 * k, win[k % (NB + 1)], win[(k + 1) % (NB + 1)]);
        if constexpr (kPlanes) load(va + 16 * MT * vp + 16 * k, wlo[k % (NB + 1)], wlo[(k + 1) % (NB + 1)]);
      };
      // Blocks 0 .. NB - 2 before the first output block.
      static_for<0, NB - 1>([&](auto kc) {
        if constexpr (decltype(kc)::value % 2 == 0) load_pair(kc);
      });
      static_for<0, kBlocks>([&](auto bc) {
        constexpr int b = decltype(bc)::value;
        if constexpr ((b + NB - 1) % 2 == 0) load_pair(std::integral_constant<int, b + NB - 1>{});
        float(&acc)[2][4] = accs[b % 2];
        static_for<0, NB>([&](auto kc) {
          constexpr int k = decltype(kc)::value;
          const uint32_t(&a)[4] = win[(b + k) % (NB + 1)];
          if constexpr (k == 0) {
            mma_f16_first(acc[0], a, wr[k][0], wr[k][1], init);
            mma_f16_first(acc[1], a, wr[k][2], wr[k][3], init);
          } else {
            if constexpr (k < NA) mma_f16(acc[0], a, wr[k][0], wr[k][1]);
            mma_f16(acc[1], a, wr[k][2], wr[k][3]);
          }
          if constexpr (kPlanes) {
            const uint32_t(&al)[4] = wlo[(b + k) % (NB + 1)];
            if constexpr (k < NA) mma_f16(acc[0], al, wrl[k][0], wrl[k][1]);
            mma_f16(acc[1], al, wrl[k][2], wrl[k][3]);
          }
        });
        // A block's results are staged behind the next block's products.
        if constexpr (b > 0) finish(accs[(b + 1) % 2], b - 1);
      });
      finish(accs[(kBlocks + 1) % 2], kBlocks - 1);
    } else {
      // Any number of steps: four output blocks at a time, a[(k + i) % 4] the
      // A operand of block b0 + k + i at step k.
      for (int b0 = 0; b0 < nblk; b0 += 4) {
        float acc[4][2][4];
        uint32_t a[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int k = 0; k < 4; ++k) acc[i][0][k] = acc[i][1][k] = init[k];
        auto load_block = [&](uint32_t (&d)[4], int blk) {
          uint32_t r0, r1;
          asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
                       : "=r"(r0), "=r"(r1)
                       : "r"(smem_addr(s.v) + (16 * m + (lane & 15)) * vp + RUN * run + 16 * blk)
                       : "memory");
          d[0] = even_bytes(r0), d[1] = even_bytes(r1), d[2] = odd_bytes(r0), d[3] = odd_bytes(r1);
        };
#pragma unroll
        for (int i = 0; i < 3; ++i) load_block(a[i], b0 + i);
        for (int k0 = 0; k0 < j.nb; k0 += 4) {
          static_for<0, 4>([&](auto kc) {
            constexpr int kk = decltype(kc)::value;
            const int k = k0 + kk;
            if (k >= j.nb) return;
            load_block(a[(kk + 3) % 4], b0 + k + 3);
            const uint4 w = wb[k * 32 + lane];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              mma_f16(acc[i][0], a[(kk + i) % 4], w.x, w.y);
              mma_f16(acc[i][1], a[(kk + i) % 4], w.z, w.w);
            }
          });
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (b0 + i < nblk) finish(acc[i], b0 + i);
      }
    }
    __syncwarp();
    const bool aligned =
        ((reinterpret_cast<uintptr_t>(j.dst) | static_cast<uintptr_t>(j.dst_stride)) & 15) == 0;
    uint8_t *const dst = j.dst + static_cast<int64_t>(y0 + 16 * m) * j.dst_stride + x0 + RUN * run;
    if (aligned && mrows == 16 && n == RUN) {
      // Whole aligned rows: the lane's 16-byte piece of every kRows-th row.
      constexpr int kRows = 32 / kBlocks;
      uint8_t *d = dst + static_cast<int64_t>(lane / kBlocks) * j.dst_stride + 16 * (lane % kBlocks);
      const uint8_t *sp = stg + lane / kBlocks * kPitch + 16 * (lane % kBlocks);
      const int64_t dstep = static_cast<int64_t>(kRows) * j.dst_stride;
#pragma unroll
      for (int row = 0; row < 16; row += kRows, d += dstep)
        if (kRows <= 16 || lane < 16 * kBlocks)
          *reinterpret_cast<uint4 *>(d) = *reinterpret_cast<const uint4 *>(sp + row * kPitch);
    } else {
      store_ragged<kBlocks>(j, stg, dst, mrows, n, lane, aligned);
    }
  }
}

// Tiles first, first + stride, ... (`count` of them) of a job: a pipeline of
// steps (all staged columns of a tile, or chunks of them where they do not
// fit), each staged into one of two buffers while the step before it is
// computed.  `taps` is cleared.
template <int NK, int NB, int NA, int MT, int W, int EPI>
__device__ __forceinline__ void mma8_tiles(const Mma8Job &j, Mma8Taps &taps, uint8_t *mem8, int first, int stride,
                                           int count) {
  using G = Mma8Geo<NK, NB, MT, W>;
  Mma8Smem s;
  s.wa = reinterpret_cast<uint32_t *>(mem8);
  s.wb = s.wa + (G::kFixed ? NK : j.nk) * 64;
  uint8_t *const raw0 = reinterpret_cast<uint8_t *>(s.wb + (G::kFixed ? NB : j.nb) * 128 * (EPI == kEpiBinomial ? 2 : 1));
  const int raw_bytes = max(G::raw_rows(j) * G::raw_pitch(j), mma8_out_bytes(mma8_run(MT, W)));
  s.raw = raw0;
  s.v = raw0 + 2 * raw_bytes;
  const int pitch = G::raw_pitch(j);
  // The current tile, the distance to the next one, and the first column of
  // the current step.
  int ty = first / j.tiles_x, tx = first - ty * j.tiles_x;
  const int dy = stride / j.tiles_x, dx = stride - dy * j.tiles_x;
  int xb = tx * W - j.hp;
  auto stage = [&](uint8_t *raw) {
    const int xe = min(tx * W + W, j.wc) + j.rc;
    stage_columns<G>(j, raw, ty * 16 * MT - j.r, min(16 * MT, j.h - ty * 16 * MT) + 2 * j.r, xb,
                     min(G::raw_cols(j), (xe - xb + 15) / 16 * 16), xe);
  };
  __syncthreads();
  spread_taps(j, taps);
  stage(s.raw);
  __syncthreads();
  build_weights<EPI>(j, taps, s.wa, s.wb);
  while (count > 0) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const int x0 = tx * W, y0 = ty * 16 * MT, cxb = xb;
    const int we = min(W, j.wc - x0), rows = min(16 * MT, j.h - y0);
    const int xe = x0 + we + j.rc;  // columns read: [x0 - rc, xe)
    const int ncols = min(G::raw_cols(j), (xe - xb + 15) / 16 * 16);
    uint8_t *const cur = s.raw;
    if (has_border_columns(j, xb, ncols, xe)) {
      fill_border_columns(j, cur, pitch, y0 - j.r, rows + 2 * j.r, xb, ncols, xe);
      __syncthreads();
    }
    // The next step's copies.
    uint8_t *const next = cur == raw0 ? raw0 + raw_bytes : raw0;
    const bool last = G::kFixed || xb + G::raw_cols(j) >= xe;
    if (last) {
      tx += dx;
      ty += dy;
      if (tx >= j.tiles_x) tx -= j.tiles_x, ++ty;
      xb = tx * W - j.hp;
      --count;
    } else {
      xb += G::raw_cols(j);
    }
    if (count > 0) stage(next);
    vertical_pass<NK, NB, MT, W, EPI>(j, s, x0, cxb, ncols);
    if (last) {
      __syncthreads();
      horizontal_pass<NK, NB, NA, MT, W, EPI>(j, s, x0, y0, we, rows);
    }
    s.raw = next;
  }
}

template <int NK, int NB, int NA, int MT, int W, int EPI>
__global__ void __launch_bounds__(kMma8Threads, 2) mma8_kernel(const __grid_constant__ Mma8Job j) {
  extern __shared__ __align__(16) uint8_t mem8[];
  __shared__ __align__(4) Mma8Taps taps;
  launch_dependents();
  clear_taps(taps);
  grid_dependency_wait();  // the source may be the previous call's output
  const int b = static_cast<int>(blockIdx.x), n = static_cast<int>(gridDim.x);
  mma8_tiles<NK, NB, NA, MT, W, EPI>(j, taps, mem8, b, n, (j.tiles_x * j.tiles_y - b + n - 1) / n);
}

// Batch plans: one launch over a table of n jobs of one instantiation, of
// which job k holds the tiles [ends[k - 1], ends[k]).  CTAs claim runs of
// `chunk` tiles through *next (0 at launch).
template <int NK, int NB, int NA, int MT, int W, int EPI>
__global__ void __launch_bounds__(kMma8Threads, 2)
    mma8_batch_kernel(const Mma8Job *__restrict__ jobs, const int *__restrict__ ends, int n, int chunk, int *next) {
  extern __shared__ __align__(16) uint8_t mem8[];
  __shared__ __align__(4) Mma8Taps taps;
  __shared__ __align__(16) Mma8Job job;
  __shared__ int claim;
  const int total = ends[n - 1];
  while (true) {
    __syncthreads();  // the last run's shared memory is dead
    if (threadIdx.x == 0) claim = atomicAdd(next, chunk);
    __syncthreads();
    int t = claim;
    if (t >= total) return;
    const int to = min(t + chunk, total);
    while (t < to) {
      int lo = 0, hi = n - 1;
      while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (ends[mid] > t) hi = mid;
        else lo = mid + 1;
      }
      __syncthreads();
      static_assert(sizeof(Mma8Job) % 4 == 0, "copied by words");
      for (int i = threadIdx.x; i < static_cast<int>(sizeof(Mma8Job) / 4); i += kMma8Threads)
        reinterpret_cast<uint32_t *>(&job)[i] = reinterpret_cast<const uint32_t *>(jobs + lo)[i];
      clear_taps(taps);
      __syncthreads();
      const int from = lo > 0 ? ends[lo - 1] : 0, count = min(to, ends[lo]) - t;
      mma8_tiles<NK, NB, NA, MT, W, EPI>(job, taps, mem8, t - from, 1, count);
      t += count;
    }
  }
}

}  // namespace kcv
