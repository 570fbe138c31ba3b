// Jobs and dispatch of the tensor-core u8 stencils (mma8.cuh).
#include <string.h>

#include <algorithm>

#include "mma8_launch.cuh"

namespace kcv {
namespace {

int round_up(int v, int a) { return (v + a - 1) / a * a; }
// Instantiations with both step counts at compile time (launch_mma8).
bool fixed_steps(const Mma8Job &j) {
  if (j.epi == kEpiArbitrary) return false;
  const int steps = 10 * j.nb + j.na;
  if (j.nk == 1) return true;  // 21, 22, 32, 33: at most 16 bytes on either side
  if (j.nk == 2) return steps == 22 || steps == 32 || steps == 33 || steps == 44 || steps == 54;
  return j.nk == 3 && (steps == 33 || steps == 43);
}

// Geometry that follows from taps, channels and the tile (j.mt, j.tile_w).
// False when the tile does not fit into shared memory.
bool shape(Mma8Job &j) {
  if (!fixed_steps(j)) j.nk = std::max(j.nk, 2);  // no instantiation for one step
  j.raw_rows = 8 * (2 * j.mt + 2 * j.nk - 1);
  j.v_cols = j.tile_w + 16 * (j.nb - 1);
  const bool fixed = fixed_steps(j);
  j.v_pitch = mma8_pitch(j.v_cols);
  j.tiles_x = (j.wc + j.tile_w - 1) / j.tile_w;
  j.tiles_y = (j.h + 16 * j.mt - 1) / (16 * j.mt);
  // 64: the last ldmatrix of a run may read one block past V.
  const int planes = j.epi == kEpiBinomial ? 2 : 1;
  const int rest = 256 * j.nk + planes * (512 * j.nb + 16 * j.mt * j.v_pitch) + 64;
  // All columns of a tile at once where two buffers of them fit, else in
  // equal chunks.
  const int cols = j.tile_w + 2 * (fixed ? mma8_round16(8 * (j.nb - 1)) : j.hp);
  for (int chunks = 1; chunks <= cols / 32; ++chunks) {
    j.raw_cols = round_up((cols + chunks - 1) / chunks, 16);
    j.raw_pitch = mma8_pitch(j.raw_cols);
    j.smem_bytes = rest + 2 * std::max(j.raw_rows * j.raw_pitch, mma8_out_bytes(mma8_run(j.mt, j.tile_w)));
    if (j.smem_bytes <= kMma8MaxSmem) return true;
  }
  return false;
}

bool plan(Mma8Job &j, int sm_count) {
  j.wc = j.w * j.c;
  j.r = j.ksize / 2;
  j.rc = j.r * j.c;
  j.hp = round_up(j.rc, 16);
  j.vo = round_up(j.rc, 4);
  j.nk = (8 + 2 * j.r + 15) / 16;
  j.nb = (j.vo + 16 + j.rc + 15) / 16;
  j.na = (j.vo + 8 + j.rc + 15) / 16;
  // Tiles of 32 rows x 256 bytes while two per SM, the resident CTAs, cover the
  // image; else 64 rows, whose halo costs half.  32 against 64 rows, 9 taps:
  // 1920x1200x1 (304 tiles of 32 rows, a full wave) 4.2 / 4.9 us, 2560x1080x1 (340)
  // 5.2 / 5.0 us, 2560x1440x1 (450) 5.9 / 5.1 us, 1366x768x3 (408) 8.9 / 7.2 us.  The least gain is at
  // 1280x720x3 (345): 5.5 / 5.4 us, and 6.5 / 6.7 us with 15 taps.
  j.tile_w = 256;
  for (j.mt = 4;; j.mt = 2) {
    if (!shape(j)) return false;
    if (j.mt == 2 || !fixed_steps(j) || static_cast<long>(j.tiles_x) * ((j.h + 31) / 32) > 2L * sm_count) return true;
  }
}

// The two-pass kernel of generic.cu reads the whole source before it writes
// (a call may filter an image in place); a tile here does not.
template <typename J>
bool overlap(const J &f, int wc) {
  const uintptr_t s0 = reinterpret_cast<uintptr_t>(f.src), d0 = reinterpret_cast<uintptr_t>(f.dst);
  const uintptr_t s1 = s0 + static_cast<uintptr_t>(f.height - 1) * f.src_stride + wc;
  const uintptr_t d1 = d0 + static_cast<uintptr_t>(f.height - 1) * f.dst_stride + wc;
  return s0 < d1 && d0 < s1;
}

template <typename J>
void common(const J &f, Mma8Job &j) {
  memset(&j, 0, sizeof(j));
  j.src = f.src;
  j.dst = f.dst;
  j.src_stride = f.src_stride;
  j.dst_stride = f.dst_stride;
  j.w = f.width;
  j.h = f.height;
  j.c = f.channels;
  j.border = f.border;
  j.border_value = f.border_value;
  j.ksize = f.ksize;
}

}  // namespace

bool mma8_job(const FilterJob &f, int sm_count, Mma8Job &j) {
  // The binomial 3x3 and 5x5 need two planes of vertical results here, and the
  // tiled stencil has cheap (constant) taps for them: it keeps the larger
  // images whose rows TMA can load.  5x5, tiled against here: 320x240x1 8.5 /
  // 3.9 us, 1920x1080x1 7.0 / 4.5 us, 1920x1080x3 9.3 / 9.9 us, 3840x2160x3 18.8
  // / 23.3 us; unaligned rows 3841x2160x1 26.3 / 14.5 us, x4 60.3 / 43.9 us.
  const bool unaligned = ((reinterpret_cast<uintptr_t>(f.src) | static_cast<uintptr_t>(f.src_stride)) & 15) != 0;
  const bool binomial = f.mode == MODE_BINOM && f.ksize <= 5 &&
                        (unaligned || static_cast<long>(f.width) * f.channels * f.height <= 4L << 20);
  if (f.mode != MODE_SIGMA && f.mode != MODE_SEP_U8 && !binomial) return false;
  common(f, j);
  for (int t = 0; t < f.ksize; ++t) {
    j.ty[t] = static_cast<uint8_t>(f.wy[t]);
    j.tx[t] = static_cast<uint8_t>(f.wx[t]);
  }
  j.epi = f.mode == MODE_SEP_U8 ? kEpiSat8 : binomial ? kEpiBinomial : kEpiRound;
  return plan(j, sm_count);
}

bool mma8_job(const GenericJob &g, int sm_count, Mma8Job &j) {
  const int wc = g.width * g.channels;
  if (overlap(g, wc)) return false;
  common(g, j);
  int sum = 0;
  for (int t = 0; t < g.ksize; ++t) {
    j.ty[t] = j.tx[t] = g.half[t <= g.ksize / 2 ? t : g.ksize - 1 - t];
    sum += j.ty[t];
  }
  j.epi = sum > 256 || (g.arbitrary && g.channels > 1) ? kEpiArbitrary : kEpiRound;
  j.saturate = g.vert_saturates;
  j.quirk = g.arbitrary && g.channels > 1;
  j.arb_border_len = g.arb_border_len;
  if (g.arbitrary && wc - 2 * g.arb_border_len >= 16) {
    j.h_sat_from = g.arb_border_len;
    j.h_sat_to = wc - g.arb_border_len;
  }
  return plan(j, sm_count);
}

namespace {

// Instantiations with both step counts at compile time.
cudaError_t launch_fixed(const Mma8Job &j, const Mma8Batch *batch, int sm_count, cudaStream_t stream) {
  if (j.epi == kEpiSat8) return launch_mma8_sat8(j, batch, sm_count, stream);
  if (j.epi == kEpiBinomial) return launch_mma8_binomial(j, batch, sm_count, stream);
  switch (mma8_batch_key(j)) {
    case 121: return launch_mma8_1_2_1(j, batch, sm_count, stream);
    case 122: return launch_mma8_1_2_2(j, batch, sm_count, stream);
    case 132: return launch_mma8_1_3_2(j, batch, sm_count, stream);
    case 133: return launch_mma8_1_3_3(j, batch, sm_count, stream);
    case 222: return launch_mma8_2_2_2(j, batch, sm_count, stream);
    case 232: return launch_mma8_2_3_2(j, batch, sm_count, stream);
    case 233: return launch_mma8_2_3_3(j, batch, sm_count, stream);
    case 244: return launch_mma8_2_4_4(j, batch, sm_count, stream);
    case 254: return launch_mma8_2_5_4(j, batch, sm_count, stream);
    case 333: return launch_mma8_3_3_3(j, batch, sm_count, stream);
    case 343: return launch_mma8_3_4_3(j, batch, sm_count, stream);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

cudaError_t launch_mma8(const Mma8Job &j, int sm_count, cudaStream_t stream) {
  if (fixed_steps(j)) return launch_fixed(j, nullptr, sm_count, stream);
  if (j.nk <= 2) return launch_mma8_2_any(j, sm_count, stream);
  return j.nk == 3 ? launch_mma8_3_any(j, sm_count, stream) : launch_mma8_0_any(j, sm_count, stream);
}

int mma8_batch_key(const Mma8Job &j) {
  if (!fixed_steps(j)) return 0;
  return 1000 * j.epi + 100 * j.nk + 10 * j.nb + j.na;
}

bool mma8_batch_job(const FilterJob &f, Mma8Job &j) { return mma8_job(f, 0, j); }

cudaError_t launch_mma8_batch(const Mma8Job &rep, const Mma8Batch &b, int sm_count, cudaStream_t stream) {
  if (b.tiles <= 0) return cudaSuccess;
  return launch_fixed(rep, &b, sm_count, stream);
}

}  // namespace kcv
