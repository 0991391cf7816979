// The choice between the filter's tile and strip kernels at sizes where one
// was at least 1.2 times as fast, measured on a B200 (148 SMs).
#include <cstdio>

#include "tm_filter_rule.h"

int main() {
  const struct {
    uint32_t W, H, C, kw, kh;
    bool strips;
  } sizes[] = {{16, 16, 3, 2, 2, false},     {64, 64, 1, 8, 32, false},   {128, 128, 1, 5, 5, false},
               {200, 150, 3, 7, 7, false},   {256, 256, 4, 8, 32, false}, {320, 240, 1, 3, 3, false},
               {512, 400, 1, 1, 1, false},   {20, 8000, 3, 2, 2, false},  {8, 40000, 3, 2, 2, false},
               {40000, 5, 4, 2, 2, false},   {1024, 768, 1, 5, 5, true},  {2048, 2048, 1, 1, 1, true},
               {2048, 2048, 3, 3, 3, true},  {4096, 4096, 1, 5, 5, true}, {4096, 4096, 4, 8, 32, true},
               {700, 500, 1, 1, 32, true},   {100, 20000, 1, 7, 7, true}, {12000, 40, 1, 8, 32, true}};
  int wrong = 0;
  for (const auto& z : sizes) {
    const uint32_t by = ipb::filter_strip_warps(z.W, z.H, z.C, z.kw, z.kh, 148);
    if ((by != 0) != z.strips || (by != 0 && by != 2 && by != 8)) {
      ++wrong;
      std::printf("%u x %u x %u, %u x %u: %u\n", z.W, z.H, z.C, z.kw, z.kh, by);
    }
  }
  return wrong;
}
