// Scalar operations of the kernels that the host can run too.
#pragma once

#include <cuda_runtime.h>
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

__host__ __device__ __forceinline__ unsigned bits_of(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  unsigned b;
  std::memcpy(&b, &x, sizeof(b));
  return b;
#endif
}
__host__ __device__ __forceinline__ float from_bits32(unsigned b) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(b);
#else
  float x;
  std::memcpy(&x, &b, sizeof(x));
  return x;
#endif
}

// FP64 <-> FP32 by integer operations where the value is in FP32's normal range (or zero): the
// conversion instructions occupy the FP64 pipe for several multiply-adds each.  Rounded to
// nearest even, as the conversions round.
__host__ __device__ __forceinline__ float narrow(double x) {
  const unsigned long long b = bits_of(x);
  const unsigned e = (unsigned)(b >> 52) & 0x7FFu, sign = (unsigned)(b >> 32) & 0x80000000u;
  if (e - 897u > 1150u - 897u) return (b << 1) == 0 ? from_bits32(sign) : (float)x;
  const unsigned long long t = (b & 0x7FFFFFFFFFFFFFFFULL) - ((unsigned long long)896 << 52);
  return from_bits32(sign | (unsigned)((t + 0x0FFFFFFFULL + ((t >> 29) & 1ULL)) >> 29));
}
__host__ __device__ __forceinline__ double widen(float x) {
  const unsigned b = bits_of(x), m = b & 0x7FFFFFFFu;
  if (m - 0x00800000u >= 0x7F000000u) return m == 0 ? from_bits((unsigned long long)b << 32) : (double)x;
  const unsigned long long t = ((unsigned long long)m << 29) + ((unsigned long long)896 << 52);
  return from_bits(t | ((unsigned long long)(b & 0x80000000u) << 32));
}
__host__ __device__ __forceinline__ float2 narrow(double2 v) { return make_float2(narrow(v.x), narrow(v.y)); }
__host__ __device__ __forceinline__ double2 widen(float2 v) { return make_double2(widen(v.x), widen(v.y)); }

// The larger of m and v (neither negative); the positive NaN, whose bits exceed all others', once
// either is one
__host__ __device__ __forceinline__ double max_or_nan(double m, double v) {
  return (m != m || v != v) ? from_bits(0x7FF8000000000000ULL) : fmax(m, v);
}

}  // namespace negf
