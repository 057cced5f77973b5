// The columns of a staged box that harmonic summing's lanes read lie inside it and hold
// the bins they stand for, for every plane and block.
#include <algorithm>
#include <cstdio>

#include "hsum_boxes.cuh"

using namespace fdas;

int main() {
  int bad = 0;
  for (int j = 2; j <= 16; ++j) {
    const int width = hs_box_width(j);
    int last = 0;
    for (int f0 = 0; f0 < 8 * j * kHsBins; f0 += kHsBins)
      for (int lane = 0; lane < 32; ++lane)
        for (int group = 0; group < 256; group += 128) {
          const int start = (f0 / j) & ~3, F = f0 + 4 * lane + group;
          // first column and how many: as the bounds read them (hs_bound_plane)
          int col, n;
          if (hs_one_value(j)) col = lane / (j / 4) + group / j, n = 1;
          else if (j == 2) col = 2 * lane + group / 2, n = 2;
          else {
            const unsigned M = 65536u / j + 1, x = f0 % j + 4 * lane + group;
            col = (int)((x * M) >> 16) + ((f0 / j) & 3);
            n = (int)(((x + 3) * M) >> 16) + ((f0 / j) & 3) - col + 1;
          }
          last = std::max(last, col + n - 1);
          for (int c = 0; c < 4; ++c) {
            const int want = (F + c) / j - start;
            if (want < col || want >= col + n) ++bad;
          }
        }
    if (last >= width || width % 4) ++bad;
    std::printf("plane %d: width %d, last column read %d\n", j, width, last);
  }
  return bad != 0;
}
