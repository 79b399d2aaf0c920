// Division by a run-time constant without the division: for n < 2^31 and 1 <= d < 2^31,
// floor(n / d) = n m >> (31 + l) with l = ceil(log2 d) and m = ceil(2^(31 + l) / d) (T.
// Granlund and P. Montgomery, "Division by invariant integers using multiplication", 1994,
// theorem 4.2: 0 <= m d - 2^(31 + l) < d <= 2^l).
#pragma once

#include <cstdint>

namespace ipeps {

struct FastDiv {
  uint32_t d = 1, m = 0x80000000u;
  int s = 31;
  FastDiv() = default;
  explicit FastDiv(uint32_t dd) : d(dd) {
    int l = 0;
    while ((uint64_t(1) << l) < d) ++l;
    s = 31 + l;
    m = uint32_t(((uint64_t(1) << s) + d - 1) / d);
  }
  __host__ __device__ __forceinline__ uint32_t div(uint32_t n) const { return uint32_t((uint64_t(n) * m) >> s); }
};

}  // namespace ipeps
