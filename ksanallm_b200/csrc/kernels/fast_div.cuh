// Division of 31-bit indices by a number that is fixed for a launch: one multiply-high and a shift instead of the dozens of
// instructions of a run-time division (a hundred for 64-bit operands), which paced kernels that find row and column of a flat index.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace ksana {

struct FastDiv {
  uint32_t d, mul, shift;
  // n / d for 0 <= n < 2^31 (round-up method: with s = ceil(log2 d) and mul = floor(2^32 (2^s - d) / d) + 1 the quotient
  // is (mulhi(n, mul) + n) >> s; the sum stays below 2^32)
  __device__ __forceinline__ uint32_t div(uint32_t n) const { return (__umulhi(n, mul) + n) >> shift; }
};

inline FastDiv make_fast_div(uint32_t d) {
  uint32_t s = 0;
  while ((1ull << s) < d) ++s;
  return FastDiv{d, static_cast<uint32_t>((((1ull << s) - d) << 32) / d + 1), s};
}

}  // namespace ksana
