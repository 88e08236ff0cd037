// sg_divide.h -- division of small numbers by a fixed divisor with one multiplication.
// Plain C++ (no CUDA types), so that host programs can check the arithmetic.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define SG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define SG_HOST_DEVICE inline
#endif

namespace sg {

// r / k = small_quotient(r, small_reciprocal(k)) for 1 <= k <= 65536 and r < 65536, k = 1
// included.  With 2^32 - 1 = m k + s, 0 <= s < k, the product (r + 1) m / 2^32 is (r + 1) / k
// less (r + 1)(1 + s) / (2^32 k), which is more than 0 and, as (r + 1) k <= 2^32, at most 1 / k:
// its floor is that of r / k.  (A reciprocal rounded up, of r itself, would be 2^32 at k = 1.)
SG_HOST_DEVICE uint32_t small_reciprocal(uint32_t k) { return 0xffffffffu / k; }
SG_HOST_DEVICE uint32_t small_quotient(uint32_t r, uint32_t reciprocal) {
    return (uint32_t)(((uint64_t)(r + 1) * reciprocal) >> 32);
}

}  // namespace sg
