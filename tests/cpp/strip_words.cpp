// Every byte that the strips' word reads touch, for narrow images at every
// alignment of their base: all must lie inside the image.
#include <cstdio>

#include "tm_strip.h"

int main() {
  using ipb::kStripRows;
  long by_words = 0, outside = 0;
  for (uint32_t base = 4; base < 8; ++base)
    for (uint32_t W = 1; W <= 12; ++W)
      for (uint32_t H = 1; H <= 7 * kStripRows; ++H)
        for (uint32_t y0 = 0; y0 < H; y0 += kStripRows) {
          if (!ipb::strip_words_inside(W, H, y0)) continue;
          ++by_words;
          const uint32_t begin = base, end = base + W * H;  // the image's addresses
          for (uint32_t r = 0; r < kStripRows; ++r)
            for (uint32_t x = 0; x < W + 4; ++x) {  // columns past the row read its last one
              const uint32_t g = base + (y0 + r) * W + (x < W ? x : W - 1), a = g & ~3u;
              outside += a < begin || a + 8 > end;
            }
        }
  std::printf("%ld strips by words, %ld reads outside\n", by_words, outside);
  return by_words > 0 && outside == 0 ? 0 : 1;
}
