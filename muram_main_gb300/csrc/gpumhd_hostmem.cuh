// Which host buffers a conversion kernel reads or writes over the link itself.
// Plain host code, which a test compiles without CUDA.
#pragma once
#include <stdint.h>

namespace hostmem {

// [p, p + bytes) lies within the one allocation or registration [start, start + size).
inline bool covers(uint64_t start, uint64_t size, uint64_t p, uint64_t bytes) {
  return p >= start && p - start <= size && bytes <= size - (p - start);
}

}  // namespace hostmem
