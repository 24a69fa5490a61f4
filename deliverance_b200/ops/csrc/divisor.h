// Division of 31-bit numbers by multiplication, for kernels whose walk over tiles would otherwise wait for a division.
#pragma once
#include <cstdint>

#include <cuda_runtime.h>

namespace dlv {

// n / d for 0 <= n < 2^31 and 1 <= d < 2^31: the high word of n * m, m = ceil(2^32 / d), is the quotient or one more. (With m d = 2^32 + e, e < d, it is
// floor(n / d + n e / (d 2^32)), whose second term is below a half.) Without the correction that is exact for n d < 2^32 only.
struct Divisor {
  unsigned d, m;  // m = 0: d is 1
  __host__ void set(int n) {
    d = static_cast<unsigned>(n < 1 ? 1 : n);
    m = d > 1 ? static_cast<unsigned>(((1ull << 32) + d - 1) / d) : 0u;
  }
  __host__ __device__ __forceinline__ int of(int n) const {
    if (m == 0u) return n;
    const unsigned u = static_cast<unsigned>(n);
#ifdef __CUDA_ARCH__
    const unsigned q = __umulhi(u, m);
#else
    const unsigned q = static_cast<unsigned>((static_cast<uint64_t>(u) * m) >> 32);
#endif
    return static_cast<int>(q * d > u ? q - 1 : q);
  }
};

}  // namespace dlv
