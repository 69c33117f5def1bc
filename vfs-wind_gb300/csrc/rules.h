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

// Columns a block of the j-line kernels takes, for lines of P chunks and blocks of
// at most max_threads.  FP32: 16, halved while the block would exceed the limit
// (8 columns for j-lines of 193..384 cells).  FP64: more, smaller blocks per SM
// measured faster (4 columns in place of 16: warm solve 31.5 -> 30.3 ms on the
// 256x192x256 towers grid); of four to eight columns, whichever leave the fewest idle
// lanes: four columns of five chunks fill 20 of a warp's 32, six fill 30.  Four
// iterations with four columns and with the rule: 192x16x192 2784 and 2372 us,
// 192x40x192 3781 and 3530, 96x40x96 1867 and 1726, 48x72x32 1044 and 1026; lines of
// 8 to 96 rows never slower.  cap > 0: no more than that many.
inline int line_columns(int P, bool fp64, int cap, int max_threads) {
  int ti = fp64 ? 4 : 16;
  if (cap > 0 && ti > cap) ti = cap;
  while (ti > 1 && ti * P > max_threads) ti >>= 1;
  if (fp64 && ti == 4) {
    auto idle = [&](int c) { return (double)((c * P + 31) / 32 * 32) / (c * P); };
    for (int c = 5; c <= 8; c++)
      if (c * P <= max_threads && (cap <= 0 || c <= cap) && idle(c) < idle(ti)) ti = c;
  }
  return ti;
}

}  // namespace vfs

#endif
