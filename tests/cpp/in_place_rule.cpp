// Rows "device ordinal start size addr bytes align gpu" on standard input; for each,
// whether a kernel of that GPU may read the range where it lies.
#include <cstdio>

#include "pointers.cuh"

int main() {
  int device, ordinal, gpu;
  unsigned long long start, size, addr, bytes, align;
  while (std::scanf("%d %d %llu %llu %llu %llu %llu %d", &device, &ordinal, &start, &size, &addr, &bytes, &align,
                    &gpu) == 8)
    std::printf("%d\n", fdas::readable_in_place(fdas::MemoryAt{device != 0, ordinal, start, size}, addr, bytes, align, gpu));
}
