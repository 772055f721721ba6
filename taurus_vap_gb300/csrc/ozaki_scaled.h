// Exact conversion of the two integer accumulators of the emulated
// products to a double: (h 2^28 + l) 2^s rounded to nearest (ties to even),
// negated when neg, with integer instructions only: the value's leading 64
// bits and whether anything follows them.
// It equals fma(double(h), 2^28, double(l)) * (+-2^s) -- both round once
// when |h|, |l| < 2^53 -- at a fraction of the cost on a part whose FP64
// pipe retires two operations per SM and cycle.  Returns false when the
// result would be subnormal or infinite (the caller then takes the
// floating-point formula, which rounds the same way there).  Plain C++ as
// well, so that host code can check it.
#pragma once

#include <cstdint>
#include <cstring>

#if defined(__CUDACC__)
#define TVAP_HD __host__ __device__ __forceinline__
#else
#define TVAP_HD inline
#endif

namespace tvap {
namespace oztc {

TVAP_HD int clz64(unsigned long long x) {
#if defined(__CUDA_ARCH__)
  return __clzll(static_cast<long long>(x));
#else
  return __builtin_clzll(x);
#endif
}

TVAP_HD double bits_to_double(unsigned long long b) {
#if defined(__CUDA_ARCH__)
  return __longlong_as_double(static_cast<long long>(b));
#else
  double d;
  std::memcpy(&d, &b, sizeof d);
  return d;
#endif
}

TVAP_HD bool scaled(long long h, long long l, int s, bool neg, double& out) {
  // hi 2^28 + lo with 0 <= lo < 2^28, then the magnitude
  constexpr unsigned kMask = (1u << 28) - 1u;
  long long hi = h + (l >> 28);
  unsigned lo = unsigned(l) & kMask;
  const bool minus = hi < 0;
  if (minus) {
    hi = ~hi + (lo == 0 ? 1 : 0);
    lo = (0u - lo) & kMask;
  }
  // its leading 64 bits, the lowest one also set for what is shifted out
  const unsigned long long uh = static_cast<unsigned long long>(hi);
  const int top = uh ? 64 - clz64(uh) : 0;
  const int sh = top > 36 ? top - 36 : 0;
  unsigned long long u = (uh << (28 - sh)) | (lo >> sh);
  u |= (lo & ((1u << sh) - 1u)) ? 1ull : 0ull;
  if (u == 0) {
    out = neg ? -0.0 : 0.0;
    return true;
  }
  const int n = clz64(u);
  const int e = 63 - n + sh + s + 1023;  // biased exponent before rounding
  if (e <= 0 || e >= 2046 || sh > 28) return false;
  // round to 53 bits: half of the last one, less one unless the last bit is
  // set; a carry out of bit 63 leaves the mantissa 0, the next power of two
  u <<= n;
  u += 0x3ffull + ((u >> 11) & 1ull);
  const unsigned long long m = (u >> 11) & ((1ull << 52) - 1ull);
  const unsigned long long up = u >> 63 ? 0ull : 1ull;
  out = bits_to_double((minus != neg ? 1ull << 63 : 0ull) | ((static_cast<unsigned long long>(e) + up) << 52) | m);
  return true;
}

}  // namespace oztc
}  // namespace tvap
