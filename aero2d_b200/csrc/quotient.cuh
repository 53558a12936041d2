// Division by a number whose reciprocal is at hand, with the bits of the division.
#pragma once
#include <cmath>
#include <cstdint>
#include <cstring>

namespace a2d {

#ifdef __CUDACC__
#define A2D_HD __host__ __device__ __forceinline__
#else
#define A2D_HD inline
#endif

// whether a - q b is exact and nothing overflows: 2^-100 <= |q| < 2^100 (FP64: 2^-960, 2^960), by the exponent
// field, one integer comparison in the chain
A2D_HD bool quotient_exact(float q) {
  uint32_t u;
  memcpy(&u, &q, sizeof u);
  return (u & 0x7fffffffu) - ((127u - 100u) << 23) < (200u << 23);
}
A2D_HD bool quotient_exact(double q) {
  uint64_t u;
  memcpy(&u, &q, sizeof u);
  return ((uint32_t)(u >> 32) & 0x7fffffffu) - ((1023u - 960u) << 20) < (1920u << 20);
}

// a / b to the bit for b in [1/2, 2^20] with y = RN(1/b): one multiplication and Markstein's correction (P.
// Markstein, IBM J. Res. Dev. 34, 1990: with q = RN(a y) and r = RN(a - q b), RN(q + r y) is
// RN(a/b)).  That wants r exact, which it is not when it falls among the subnormals: there,
// and for infinities and NaN, the division itself.  A zero is a y, sign and all.
template <typename T>
A2D_HD T quotient(T a, T b, T y) {
  using std::fma;
  const T q = a * y;
  const T r = fma(-q, b, a);
  if (quotient_exact(q)) return fma(r, y, q);
  return a == T(0) ? q : a / b;
}

}  // namespace a2d
