// Which memory of a caller's the kernels may read where it lies (plain C++: the
// rule is host code).
#pragma once
#include <cstddef>
#include <cstdint>

namespace fdas {

// What the driver knows about an address.
struct MemoryAt {
  bool device;           // plain device memory (not managed, not host, not unknown)
  int ordinal;           // of the GPU that holds it
  uint64_t start, size;  // the allocation around it; size 0: unknown
};

// A kernel of GPU `device` may read `bytes` at `addr` itself.  A copy takes memory of
// any GPU, of any alignment, and refuses a range that leaves its allocation; a kernel
// that reads another GPU's memory without peer access, or past the end, loses the
// context, so whatever is not known to be this GPU's own goes through the copy.
inline bool readable_in_place(const MemoryAt &m, uint64_t addr, uint64_t bytes, uint64_t align, int device) {
  return m.device && m.ordinal == device && addr % align == 0 && m.start <= addr && bytes <= m.size &&
         addr - m.start <= m.size - bytes;
}

}  // namespace fdas
