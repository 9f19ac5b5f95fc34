// Which host buffers a conversion kernel reads or writes over the link itself.
// Plain host code, which a test compiles without CUDA.
#pragma once
#include <stdint.h>

namespace hostmem {

// [p, p + bytes) lies within the one allocation or registration [start, start + size).
inline bool covers(uint64_t start, uint64_t size, uint64_t p, uint64_t bytes) {
  return p >= start && p - start <= size && bytes <= size - (p - start);
}

// Whether a kernel moves records of nf values of `size` bytes at this (pinned)
// address over the link itself: single values, which are contiguous, and records
// of eight in 16-byte pieces.  Unaligned records move value by value, a record
// per thread, which only the upload of floats takes well.  128 x 384 x 384,
// directly and through the staging buffer, ms: download of doubles 65.7, 6.9, of
// floats 22.0, 3.5; upload of doubles 12.1, 6.9, of floats 3.1, 3.6 (aligned,
// directly: 6.6, 3.3; 6.1, 3.0).
inline bool moves_directly(int nf, int size, uint64_t address, bool download) {
  if (nf == 1) return true;
  return nf == 8 && (address % 16 == 0 || (size == 4 && !download));
}

}  // namespace hostmem
