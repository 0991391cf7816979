// tm_strip.h -- where the integral image's strips may be read by words. Plain
// C++ beside the kernel, so that the bound is checked on the host.
#pragma once
#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define IPB_HOST_DEVICE __host__ __device__
#else
#define IPB_HOST_DEVICE
#endif

namespace ipb {

constexpr uint32_t kStripRows = 16;  // image rows per strip

// Whether rows [y0, y0 + 16) of a W x H byte image, read four bytes from any
// column as the two aligned words around them (at most 3 bytes before the
// first one, 7 past the row's last), stay inside the image: up to seven bytes,
// not one row, must follow the strip, and narrow rows are shorter than that.
IPB_HOST_DEVICE constexpr bool strip_words_inside(uint32_t W, uint32_t H, uint32_t y0) {
  return y0 != 0 && H - y0 > kStripRows && (size_t)(H - y0 - kStripRows) * W >= 7;
}

}  // namespace ipb
