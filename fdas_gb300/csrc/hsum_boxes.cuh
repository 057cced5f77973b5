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

// Plane j's box holds the values at the bins f0 / j .. (f0 + kHsBins - 1) / j of a block
// from f0, its first column at (f0 / j) & ~3.  Its columns (a multiple of 4: 16-byte rows)
// are the most that any block takes (the shift of f0 / j against the box's start repeats
// every 4 j blocks); nothing is read past them.
FDAS_HD constexpr int hs_box_width(int j) {
  int width = 0;
  for (int f0 = 0; f0 < 4 * j * kHsBins; f0 += kHsBins) {
    const int w = (f0 + kHsBins - 1) / j + 1 - ((f0 / j) & ~3);
    if (w > width) width = w;
  }
  return (width + 3) & ~3;
}
// Planes whose blocks start on a column of their own, and where the four bins of a
// lane's group share one value: read at offsets known to the compiler.
FDAS_HD constexpr bool hs_one_value(int j) { return kHsBins % j == 0 && j % 4 == 0; }

}  // namespace fdas
