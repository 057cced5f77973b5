// Box shapes of harmonic summing's staging, host and device (plain C++ but for the
// decorations).
#pragma once

#ifdef __CUDACC__
#define FDAS_HD __host__ __device__
#else
#define FDAS_HD
#endif

namespace fdas {

constexpr int kHsBins = 256;  // spectrum bins per harmonic-summing work item

// Plane j's box holds the values of the bins f0 / j .. (f0 + kHsBins - 1) / j of a block
// from f0, its first column at (f0 / j) & ~3.  Where j divides kHsBins and 4 divides j,
// the four bins of a lane's group share one value; where j only divides kHsBins
// (j = 2) they are two aligned ones.  In both cases the block's values are aligned and
// kHsBins / j.  For the other planes a group takes values at two neighbouring columns,
// of which the second may be one past the last bin's.
FDAS_HD constexpr bool hs_aligned(int j) { return kHsBins % j == 0; }
FDAS_HD constexpr bool hs_one_value(int j) { return hs_aligned(j) && j % 4 == 0; }

// Columns of plane j's box (a multiple of 4: 16-byte rows): the last column that the
// kernel reads, that of bin F / j + 1 of the last lane's group, for any block of f0 (the shift
// of f0 / j against the box's start repeats every 4 j blocks).
FDAS_HD constexpr int hs_box_width(int j) {
  int width = kHsBins / j;
  if (!hs_aligned(j))
    for (int f0 = 0; f0 < 4 * j * kHsBins; f0 += kHsBins) {
      const int w = (f0 + kHsBins - 4) / j + 2 - ((f0 / j) & ~3);
      if (w > width) width = w;
    }
  return (width + 3) & ~3;
}

}  // namespace fdas
