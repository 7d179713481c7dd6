// Scalar operations of the kernels that the host can run too.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

namespace negf {

__host__ __device__ __forceinline__ unsigned long long bits_of(double x) {
#ifdef __CUDA_ARCH__
  return (unsigned long long)__double_as_longlong(x);
#else
  unsigned long long b;
  std::memcpy(&b, &x, sizeof(b));
  return b;
#endif
}
__host__ __device__ __forceinline__ double from_bits(unsigned long long b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  std::memcpy(&x, &b, sizeof(x));
  return x;
#endif
}

// The larger of m and v (neither negative); the positive NaN, whose bits exceed all others', once
// either is one
__host__ __device__ __forceinline__ double max_or_nan(double m, double v) {
  return (m != m || v != v) ? from_bits(0x7FF8000000000000ULL) : fmax(m, v);
}

}  // namespace negf
