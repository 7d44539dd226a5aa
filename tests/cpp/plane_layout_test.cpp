// The plane updates name no word past a sketch when they bring its columns to L2
// (graphzeppelin_b200/csrc/gz_plane_layout.h): every geometry of 18 to 256 columns and 1 to 63 buckets.
#include <cstdio>

#include "gz_plane_layout.h"

int main() {
  int bad = 0;
  for (uint32_t C = 18; C <= 256; ++C)
    for (uint32_t B = 1; B <= 63; ++B) {
      const uint32_t words = 3 * (C * B + 1);
      for (uint32_t c = 0; c < C; ++c) {
        const uint32_t at = 3 * c * B + gz::column_second_word(B);
        bad += at >= words || at >= 3 * (c + 1) * B;
      }
    }
  if (!bad) std::printf("plane layout ok\n");
  return bad != 0;
}
