// Smallest and largest value of a map: order-preserving keys and a CTA's share.
#pragma once
#include <cuda_runtime.h>

namespace sred {

// Order-preserving key of a float (-0 below +0), and back.
__device__ __forceinline__ unsigned ord_bits(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord_float(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// A CTA's smallest and largest key into mm (all threads of the CTA call it).
__device__ __forceinline__ void cta_minmax(unsigned lo, unsigned hi, unsigned* mm) {
  __shared__ unsigned s_lo[8], s_hi[8];  // 256 threads
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if ((threadIdx.x & 31) == 0) {
    s_lo[threadIdx.x >> 5] = lo;
    s_hi[threadIdx.x >> 5] = hi;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    lo = __reduce_min_sync(0xffffffffu, s_lo[threadIdx.x & 7]);
    hi = __reduce_max_sync(0xffffffffu, s_hi[threadIdx.x & 7]);
    if (threadIdx.x == 0 && lo <= hi) {
      atomicMin(mm, lo);
      atomicMax(mm + 1, hi);
    }
  }
}

}  // namespace sred
