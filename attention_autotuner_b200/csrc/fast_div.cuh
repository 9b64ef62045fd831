// Division of a non-negative int by a launch constant, as the high word of one product; also compiled for the host by its test.
#pragma once

#include <stdint.h>

namespace ab200 {

#ifdef __CUDACC__
#define AB200_BOTH __host__ __device__ __forceinline__
#else
#define AB200_BOTH inline
#endif

// n / d for 0 <= n < 2^31 and 1 <= d < 2^31. With s = ceil(log2 d) and mul = ceil(2^(31 + s) / d) the product
// n mul / 2^(31 + s) exceeds n / d by less than n / 2^(31 + s) <= 1 / d, so that no integer lies between the two; mul is below
// 2^32 because d > 2^(s - 1).
struct FastDiv {
  uint32_t mul, shift;
};
inline FastDiv make_fast_div(int d) {
  uint32_t s = 0;
  while ((1ull << s) < static_cast<uint32_t>(d)) ++s;
  return FastDiv{static_cast<uint32_t>(((1ull << (31 + s)) + d - 1) / d), s};
}
AB200_BOTH int fast_div(int n, FastDiv d) {
  const uint32_t n2 = static_cast<uint32_t>(n) << 1;
#ifdef __CUDA_ARCH__
  return static_cast<int>(__umulhi(n2, d.mul) >> d.shift);
#else
  return static_cast<int>(static_cast<uint32_t>((static_cast<uint64_t>(n2) * d.mul) >> 32) >> d.shift);
#endif
}

}  // namespace ab200
