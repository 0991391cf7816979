// tm_filter_rule.h -- which of the two shared-memory kernels of tm_filter.cu
// takes an image and kernel size. Plain C++ beside the kernels, so that the
// choice is checked on the host.
#pragma once
#include <cstdint>

#include "tm_strip.h"

namespace ipb {

// A block of the tile kernel: 32 x 8 pixels, one per thread.
constexpr uint32_t kFilterTileW = 32, kFilterTileH = 8;
// A block of the strip kernel: 128 elements by 8 or 32 rows, 4 x 4 elements
// per thread.
constexpr uint32_t kFilterStripW = 128, kFilterStripRows = 4;

// Elements staged ahead of a strip: the leftmost tap's, rounded up to a word.
IPB_HOST_DEVICE constexpr uint32_t filter_strip_pad(uint32_t C, uint32_t kw) { return ((kw / 2) * C + 3) & ~3u; }
// Staged elements per row: the strip, the pad and the taps to the right.
IPB_HOST_DEVICE constexpr uint32_t filter_strip_pitch(uint32_t C, uint32_t kw) {
  return filter_strip_pad(C, kw) + ((kFilterStripW + (kw - 1 - kw / 2) * C + 3) & ~3u);
}

// Estimated microseconds, fitted to 3960 device times of each kernel (images
// of 16 x 16 to 4000 x 2500, shallow and narrow ones, 1, 3 and 4 channels,
// kernels of 1 x 1 to 8 x 32): a launch and the longest thread's work, and per
// block on an SM its staging and taps.
inline double filter_tile_cost(uint32_t W, uint32_t H, uint32_t C, uint32_t kw, uint32_t kh, uint32_t sms) {
  const double blocks = (double)((W + kFilterTileW - 1) / kFilterTileW) * ((H + kFilterTileH - 1) / kFilterTileH);
  const double taps = (double)C * kw * kh;
  return 1.9 + 0.07 * kh + 0.007 * taps + blocks / sms * (0.16 + 0.021 * kh + 0.0057 * taps);
}
// by: warps per block, each of four rows.
inline double filter_strip_cost(uint32_t W, uint32_t H, uint32_t C, uint32_t kw, uint32_t kh, uint32_t by,
                                uint32_t sms) {
  const uint32_t rows = kFilterStripRows * by;
  const double n = (double)W * C, gx = (double)(((uint64_t)W * C + kFilterStripW - 1) / kFilterStripW);
  const double blocks = gx * ((H + rows - 1) / rows), taps = (double)kw * kh;
  const double pitch = filter_strip_pitch(C, kw), staged = (rows + kh - 1.0) * pitch / 4;
  const double clamped = (rows + kh - 1.0) * (pitch - n / gx) / 4;  // words past the row's ends, by bytes
  return 2.4 + 0.19 * staged / (32 * by) + 0.036 * taps +
         blocks / sms * (0.0175 * (staged + clamped) / 32 + 0.0042 * by * taps);
}

// Warps per block of the strip kernel, 2 or 8, or 0 for the tile kernel. The
// tile kernel always where its blocks are at most two per SM: they all run at
// once, and its threads have a sixteenth of the outputs (128 x 128, 5 x 5: 2.4
// against 4.2 us; 4096 x 4096: 209 and 56). Over the timed sizes the choice is
// 1 % slower than the faster kernel on average; strips for all were 16 %.
inline uint32_t filter_strip_warps(uint32_t W, uint32_t H, uint32_t C, uint32_t kw, uint32_t kh, uint32_t sms) {
  const uint64_t blocks = (uint64_t)((W + kFilterTileW - 1) / kFilterTileW) * ((H + kFilterTileH - 1) / kFilterTileH);
  if (blocks <= 2ull * sms) return 0;
  const double few = filter_strip_cost(W, H, C, kw, kh, 2, sms), many = filter_strip_cost(W, H, C, kw, kh, 8, sms);
  const uint32_t by = few < many ? 2u : 8u;
  return filter_tile_cost(W, H, C, kw, kh, sms) < (by == 2 ? few : many) ? 0u : by;
}

}  // namespace ipb
