// rules.h -- decisions about a call that need no device (plain C++, checked without one).
#ifndef VFS_RULES_H
#define VFS_RULES_H

#include <cstdint>

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

}  // namespace vfs

#endif
