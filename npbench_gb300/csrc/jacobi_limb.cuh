// Binary64 Jacobi-2D rows in binary32 limbs (fxl.cuh); the point arithmetic and its
// order are jacobi_core.cuh's.
//
// A warp loads 32 adjacent columns and owns the 30 inner ones; it walks down two
// row ranges at once, rows i and i + half in the two halves of each packed
// operation, so that every neighbour of a pair is a pair.  Rows i-1, i, i+1 stay
// in registers as limbs, each converted once; west and east come by shuffle.
// Additions and the product by 0.2 run in limbs (about 100 instructions a point, 105
// with the product on the integer pipes, against 137 of the fixed-point strips).
//
// The frame of a strip follows the largest value of its first row.  Points that limbs
// leave open (fxl::fifth_of), among them any with an input out of the frame, are
// evaluated in hardware binary64 from memory; a strip with more than eight values out
// of the frame in its first rows (negative ones, say) takes hardware binary64
// throughout, but for the product: standard normal values at 1000^2, TSTEPS=50, 1.24 ms,
// 1.41 with it on the binary64 pipe (the fixed-point strips 1.38); 600 x 2000, 30, 0.84,
// 0.96 and 0.91; 2800^2, 11, 1.47, 1.78 and 1.82.
#pragma once

#include "fxl.cuh"
#include "jacobi_core.cuh"

namespace npbgb {
namespace jlimb {

constexpr int kStrip = 30;  // columns a warp writes

using fxl::L3;
using fxl::P2;

__device__ __forceinline__ double hardware(double c, double w, double e, double s, double n) {
  return mul_rn(0.2, add_rn(add_rn(add_rn(add_rn(c, w), e), s), n));
}
// CG here and below: loads go through the L2, for arrays that other CTAs of the same launch
// write.
template <bool CG>
__device__ __forceinline__ double load(const double* p) {
  if constexpr (CG) return __ldcg(p); else return *p;
}
template <bool CG>
static __device__ __noinline__ double hardware_point(const double* p, int64_t nx) {
  return hardware(load<CG>(p), load<CG>(p - 1), load<CG>(p + 1), load<CG>(p + nx), load<CG>(p - nx));
}

// The two arithmetics of a pair.
struct Limbs {
  using Pair = L3;
  fxl::Consts K;
  P2 t, c;
  bool sure_a, sure_b;
  __device__ __forceinline__ Pair from(double a, double b) const {
    return fxl::from_f64(K, static_cast<uint64_t>(__double_as_longlong(a)),
                         static_cast<uint64_t>(__double_as_longlong(b)));
  }
  static __device__ __forceinline__ P2 up1(P2 a) {  // from the lane to the west
    return fxl::pair(__shfl_up_sync(0xffffffffu, fxl::first(a), 1), __shfl_up_sync(0xffffffffu, fxl::second(a), 1));
  }
  static __device__ __forceinline__ P2 down1(P2 a) {
    return fxl::pair(__shfl_down_sync(0xffffffffu, fxl::first(a), 1),
                     __shfl_down_sync(0xffffffffu, fxl::second(a), 1));
  }
  __device__ __forceinline__ void point(const Pair& x, const Pair& s, const Pair& n, double& va, double& vb) {
    L3 a = fxl::add(x, L3{up1(x.h), up1(x.m), up1(x.l)});
    fxl::round_pos(K, a);
    a = fxl::add(a, L3{down1(x.h), down1(x.m), down1(x.l)});
    fxl::round_pos(K, a);
    a = fxl::add(a, s);
    fxl::round_pos(K, a);
    a = fxl::add(a, n);
    fxl::round_pos(K, a, t);
    const fxl::Words w = fxl::words_of(K, fxl::fifth_of(K, a, t, sure_a, sure_b, c));
    va = __longlong_as_double(static_cast<long long>(fxl::to_f64<59>(
        fxl::first(w.h), fxl::first(w.m), fxl::first(w.l), fxl::first(c), K.scale + fxl::kFifthScale)));
    vb = __longlong_as_double(static_cast<long long>(fxl::to_f64<59>(
        fxl::second(w.h), fxl::second(w.m), fxl::second(w.l), fxl::second(c), K.scale + fxl::kFifthScale)));
  }
};
struct Hardware {
  struct Pair { double a, b; };
  __device__ __forceinline__ Pair from(double a, double b) const { return Pair{a, b}; }
  __device__ __forceinline__ void point(const Pair& x, const Pair& s, const Pair& n, double& va, double& vb) const {
    const Pair w{__shfl_up_sync(0xffffffffu, x.a, 1), __shfl_up_sync(0xffffffffu, x.b, 1)};
    const Pair e{__shfl_down_sync(0xffffffffu, x.a, 1), __shfl_down_sync(0xffffffffu, x.b, 1)};
    const double a = add_rn(add_rn(add_rn(add_rn(x.a, w.a), e.a), s.a), n.a);
    const double b = add_rn(add_rn(add_rn(add_rn(x.b, w.b), e.b), s.b), n.b);
    // The product on the integer pipes leaves four operations of five on the binary64
    // pipe.  For the whole warp or not at all: predicated, the other one would be issued
    // too.
    if (__all_sync(0xffffffffu, fx::mul02_is_normal(a) && fx::mul02_is_normal(b))) {
      va = fx::mul02_normal(a);
      vb = fx::mul02_normal(b);
    } else {
      va = mul_rn(0.2, a);
      vb = mul_rn(0.2, b);
    }
  }
};

// The upper word of a finite value that is not negative, or 0.
__device__ __forceinline__ uint32_t finite_word(double x) {
  const uint32_t hi = static_cast<uint32_t>(__double2hiint(x));
  return hi < 0x7ff00000u ? hi : 0u;
}

// Output rows [r0, r1) at columns k0 .. k0 + 29 (warp-collective).  False, and nothing
// written, if M is Limbs and the strip wants Hardware.
template <class M, bool CG = false>
__device__ __forceinline__ bool rows(M m, const double* __restrict__ src, double* __restrict__ dst, int64_t nx,
                                     int64_t k0, int64_t r0, int64_t r1) {
  using Pair = typename M::Pair;
  constexpr bool kLimbs = sizeof(Pair) == sizeof(L3);
  const int lane = threadIdx.x & 31;
  const int64_t j = k0 - 1 + lane;
  const bool in = j < nx;
  const bool out = lane >= 1 && lane <= kStrip && j < nx - 1;
  const int count = int(r1 - r0), half = (count + 1) >> 1;
  const int64_t apart = int64_t(half) * nx;
  const double* p = src + (r0 - 1) * nx + j;
  double* o = dst + r0 * nx + j;
  // Row r0 - 1 + q of the first range and of the second (which may be one short:
  // its last row is then read twice and not written).
  int q = 0;
  double ra, rb;
  const bool odd = (count & 1) != 0;
  auto next = [&]() {
    ra = in ? load<CG>(p) : 0.0;
    rb = in ? load<CG>(p + (odd && q > half ? apart - nx : apart)) : 0.0;
    p += nx;
    ++q;
  };
  next();
  const double za = ra, zb = rb;
  next();
  if constexpr (kLimbs) {
    const uint32_t wa = finite_word(ra), wb = finite_word(rb);
    m.K.scale = fxl::frame_of(__reduce_max_sync(0xffffffffu, wa > wb ? wa : wb));
  }
  Pair x0 = m.from(za, zb), x1 = m.from(ra, rb), x2;
  next();
  if constexpr (kLimbs) {
    const bool lost = fxl::refused_value(x0) || fxl::refused_value(x1);
    if (__popc(__ballot_sync(0xffffffffu, lost)) > 8) return false;
  }
  int i = 0;
  auto step = [&](const Pair& xp, const Pair& xc, Pair& xn) -> bool {
    xn = m.from(ra, rb);
    if (i + 1 < half) next();
    double va, vb;
    m.point(xc, xn, xp, va, vb);
    const bool second = i + half < count;
    if constexpr (kLimbs) {
      if (!(m.sure_a && m.sure_b)) {
        const double* at = src + (o - dst);
        // the limbs of a zero sum's product are zero
        if (!m.sure_a) va = out && fxl::first(m.t) != 0u ? hardware_point<CG>(at, nx) : 0.0;
        if (!m.sure_b) vb = out && second && fxl::second(m.t) != 0u ? hardware_point<CG>(at + apart, nx) : 0.0;
      }
    }
    if (out) {
      o[0] = va;
      if (second) o[apart] = vb;
    }
    o += nx;
    return ++i < half;
  };
  while (step(x0, x1, x2) && step(x1, x2, x0) && step(x2, x0, x1)) {
  }
  return true;
}

template <bool CG = false>
static __device__ __noinline__ void rows_hardware(const double* __restrict__ src, double* __restrict__ dst, int64_t nx,
                                                  int64_t k0, int64_t r0, int64_t r1) {
  rows<Hardware, CG>(Hardware{}, src, dst, nx, k0, r0, r1);
}

}  // namespace jlimb
}  // namespace npbgb
