// rules.h -- decisions about a call that need no device (plain C++, checked without one).
#ifndef VFS_RULES_H
#define VFS_RULES_H

#include <cstddef>
#include <cstdint>
#include <initializer_list>

namespace vfs {

// Whether kernels of a handle on device `device` may work on a caller's FP64
// array where it lies: memory of that device or managed memory, at an address
// whose elements are aligned.  Everything else (host memory, another device's
// memory, which a kernel cannot reach without peer access) goes through the
// handle's staging copies, which take any address.
enum class MemoryType { host, device, managed };
inline bool in_place(MemoryType type, int memory_device, int device, uintptr_t address) {
  if (address % sizeof(double)) return false;
  return type == MemoryType::managed || (type == MemoryType::device && memory_device == device);
}

// Whether two of a call's arrays share a byte (a null one shares none).  The
// stages that update arrays in place read one array's neighbours while they write
// another: arrays that overlap are staged, as all were once, so that every value is
// formed from the arrays as they were passed.
struct Span {
  const void *p;
  size_t bytes;
};
inline bool overlap(std::initializer_list<Span> spans) {
  for (const Span &a : spans)
    for (const Span &b : spans) {
      if (&a == &b || !a.p || !b.p) continue;
      const uintptr_t x = (uintptr_t)a.p, y = (uintptr_t)b.p;
      if (x < y + b.bytes && y < x + a.bytes) return true;
    }
  return false;
}

}  // namespace vfs

#endif
