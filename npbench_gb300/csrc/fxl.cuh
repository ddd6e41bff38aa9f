// Exact binary64 addition in fixed point held as three binary32 limbs, two
// values at a time on the packed binary32 instructions.
//
// fx64.cuh keeps a value as one 64-bit integer and rounds it on the integer
// ALU, about twelve instructions an addition.  GB300 measures 60 packed f32x2
// operations (120 binary32) per SM and clock against 60 shifts or logic
// operations and 1.6 binary64 additions, so the same exact arithmetic costs
// about half as many issue slots when the value is the sum of three binary32
// numbers on fixed grids:
//
//   x = h + m + l,   h a multiple of 2^-20, 0 <= m < 2^-20 a multiple of 2^-40,
//                    0 <= l < 2^-40 a multiple of 2^-59
//
// for x == +0 or x in [2^-7, 1), i.e. every binary64 whose unit in the last
// place is at least 2^-59 (frame 59 of fx64.cuh, 20 + 20 + 19 bits).  h and m
// are stored times 2^8, l times 2^37 (see round_any), which makes every grid
// step, bound and exponent below a power-of-two multiple of the one stated.
//
// Sums.  Limbs add separately, with no carry between them.  As long as the
// weights of the inputs in a sum add up to at most 16 in h and 16 in m and l
// (Heat-3D's 14 and 12, Jacobi-2D's 5), every limb stays an integer multiple of
// its grid step below 2^24 steps, so all limb additions and products by small
// integers are exact.
//
// Rounding.  For an exact sum T = h + m + l with 2^e <= |T| < 2^(e+1), IEEE
// rounds to a multiple of u = 2^(e-52), ties to even.  Frame 59 holds T exactly,
// so nothing is rounded for e < -6; for -6 <= e <= 3, u <= 2^-49 divides h and
// m with an even quotient, and rounding T means rounding l to a multiple of u,
// ties to even: l' = (l + C) - C for a binary32 C whose unit in the last place
// is u, i.e. C in [2^(e-29), 2^(e-28)), as long as l + C stays in that binade.
// l is stored times 2^29 more than h, so that C is the power of two 2^e of the
// sum itself: the sum's binary32 approximation t with its mantissa cleared.
//
//   round_pos (all inputs added with positive sign): r = m + l and t = h + r,
//   both rounded toward zero.  Truncation is monotone and every power of two
//   2^k >= 2^-20 leaves D = 2^k - h exactly representable, so t >= 2^k if and
//   only if T >= 2^k: t has T's exponent.  0 <= l < 2^-37.7 keeps l + C inside
//   the binade of C = 2^e.
//
//   round_any (signed sums): t1 = fl(h + m), its exact error m - (t1 - h)
//   (Fast2Sum; where |h| < |m| both are so small that t1 is exact), and
//   r = fl(error + l), whose sign is exact.  |r| is below one unit of t1, so T
//   lies in t1's binade unless t1 is a power of two and r has the other sign,
//   which is what t = t1 + r rounded toward zero gives.  With a signed l the
//   constant is C = 2^e + 2^-8 (in l's scale): l > -2^-8 cannot leave the
//   binade below, and where nothing may be rounded (e < -6) C >= 2^-8 keeps
//   l + C exact: all three are multiples of 2^-30 below 2^-6, or C is 2^-8 plus
//   at most one unit and l + C is below 2^-7.
//
// A value outside the range carries h = NaN, which every sum and t inherit; the
// caller tests t once at the end.  Results are +0 or positive there (a zero sum
// has t = 0).
//
// The header compiles for the device and for the host; the host build
// (rounding toward zero through fesetround) is checked against the CPU's
// IEEE binary64.
#pragma once

#include <cstdint>
#include <cmath>
#include <cstring>

#include "fx64.cuh"

#if !defined(__CUDA_ARCH__)
#include <cfenv>
#endif

namespace npbgb {
namespace fxl {

// Two binary32 numbers, the first in the low half.
struct P2 {
  uint64_t v;
};

// The limbs of two values.
struct L3 {
  P2 h, m, l;
};

NPBGB_FX_FN P2 pair(uint32_t a, uint32_t b) {
#if defined(__CUDA_ARCH__)
  P2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "r"(a), "r"(b));
  return r;
#else
  return P2{static_cast<uint64_t>(b) << 32 | a};
#endif
}
NPBGB_FX_FN uint32_t first(P2 a) { return static_cast<uint32_t>(a.v); }
NPBGB_FX_FN uint32_t second(P2 a) { return static_cast<uint32_t>(a.v >> 32); }
NPBGB_FX_FN P2 both(uint32_t a) { return pair(a, a); }

#if !defined(__CUDA_ARCH__)
inline float f32_of(uint32_t b) {
  float f;
  std::memcpy(&f, &b, 4);
  return f;
}
inline uint32_t bits32(float f) {
  uint32_t b;
  std::memcpy(&b, &f, 4);
  return b;
}
template <typename F>
inline P2 each(P2 a, P2 b, P2 c, F f) {
  return pair(bits32(f(f32_of(first(a)), f32_of(first(b)), f32_of(first(c)))),
              bits32(f(f32_of(second(a)), f32_of(second(b)), f32_of(second(c)))));
}
// One operation toward zero (the volatiles keep it between the mode changes).
template <typename F>
inline float toward_zero(float a, float b, float c, F f) {
  volatile float x = a, y = b, z = c;
  std::fesetround(FE_TOWARDZERO);
  volatile float r = f(x, y, z);
  std::fesetround(FE_TONEAREST);
  return r;
}
#endif

NPBGB_FX_FN P2 add(P2 a, P2 b) {
#if defined(__CUDA_ARCH__)
  P2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
#else
  return each(a, b, b, [](float x, float y, float) { return x + y; });
#endif
}
NPBGB_FX_FN P2 add_rz(P2 a, P2 b) {
#if defined(__CUDA_ARCH__)
  P2 r;
  asm("add.rz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
#else
  return each(a, b, b, [](float x, float y, float z) {
    return toward_zero(x, y, z, [](float p, float q, float) { return p + q; });
  });
#endif
}
// a * b + c with one rounding.  Differences are written as multiply-adds by minus
// one, which take a constant operand the kernels hold anyway.
NPBGB_FX_FN P2 fma(P2 a, P2 b, P2 c) {
#if defined(__CUDA_ARCH__)
  P2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
#else
  return each(a, b, c, [](float x, float y, float z) { return std::fma(x, y, z); });
#endif
}
NPBGB_FX_FN P2 fma_rz(P2 a, P2 b, P2 c) {
#if defined(__CUDA_ARCH__)
  P2 r;
  asm("fma.rz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
#else
  return each(a, b, c, [](float x, float y, float z) {
    return toward_zero(x, y, z, [](float p, float q, float s) { return std::fma(p, q, s); });
  });
#endif
}

NPBGB_FX_FN L3 add(const L3& a, const L3& b) { return L3{add(a.h, b.h), add(a.m, b.m), add(a.l, b.l)}; }
// a + k * b, k a pair of small integers (exact)
NPBGB_FX_FN L3 fma(P2 k, const L3& b, const L3& a) {
  return L3{fma(k, b.h, a.h), fma(k, b.m, a.m), fma(k, b.l, a.l)};
}

// Binary32 patterns: the values whose units are the grid steps, and factors.
constexpr uint32_t kHBase = 0x45000000u;   // 2^11, unit 2^-12 = 2^8 * 2^-20
constexpr uint32_t kMBase = 0x3b000000u;   // 2^-9, unit 2^-32 = 2^8 * 2^-40
constexpr uint32_t kLBase = 0x40200000u;   // 2.5, unit 2^-22 = 2^37 * 2^-59 (room below zero and above one)
constexpr uint32_t kOne = 0x3f800000u;     // 1 = 2^37 * 2^-37, the 2^-8 of round_any in l's scale
constexpr uint32_t kLtoM = 0x31000000u;    // 2^-29
constexpr uint32_t kSign = 0x80000000u;
constexpr uint64_t kExpBoth = 0x7f8000007f800000ull;
constexpr uint32_t kNaN = 0x7fffffffu;

// The constants as register operands.  The packed instructions take no
// immediates; made opaque once per kernel, they stay in registers instead of
// being rebuilt (two moves) at every use.
struct Consts {
  P2 h_base, m_base, l_base, one, minus_one, l_to_m, h_scale, minus_two, eight;
  P2 fifth, minus_five, m_to_l, t_to_l, z_scale, third;  // (fifth_of)
  uint32_t implicit, half_bit;
  uint32_t scale = 0;  // the frame holds x * 2^-s: s << 20 (frame_of)
};
NPBGB_FX_FN uint32_t opaque(uint32_t v) {
#if defined(__CUDA_ARCH__)
  uint32_t r;
  asm volatile("mov.b32 %0, %1;" : "=r"(r) : "r"(v));
  return r;
#else
  return v;
#endif
}
NPBGB_FX_FN P2 opaque_both(uint32_t v) { return pair(opaque(v), opaque(v)); }
NPBGB_FX_FN Consts consts() {
  Consts k;
  k.h_base = opaque_both(kHBase);
  k.m_base = opaque_both(kMBase);
  k.minus_one = opaque_both(kOne | kSign);
  k.l_base = opaque_both(kLBase);
  k.one = opaque_both(kOne);
  k.l_to_m = opaque_both(kLtoM);
  k.h_scale = opaque_both(0x83800000u);  // -2^-120
  k.minus_two = opaque_both(0xc0000000u);
  k.eight = opaque_both(0x41000000u);
  k.fifth = opaque_both(0x3e4cccccu);       // just below 1/5
  k.minus_five = opaque_both(0xc0a00000u);
  k.m_to_l = opaque_both(0x4e000000u);      // 2^29
  k.t_to_l = opaque_both(0x33000000u);      // 2^-25
  k.z_scale = opaque_both(0x49cccccdu);     // 2^23 / 5
  k.third = opaque_both(0x3eaaaa80u);       // (1 - 2^-18) / 3
  k.half_bit = opaque(0x400000u);
  k.implicit = opaque(0x100000u);
  return k;
}

NPBGB_FX_FN uint32_t shf_l(uint32_t lo, uint32_t hi, uint32_t s) {  // high word of hi:lo << (s % 32)
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(lo, hi, s);
#else
  return static_cast<uint32_t>(((static_cast<uint64_t>(hi) << 32 | lo) << (s & 31u)) >> 32);
#endif
}
NPBGB_FX_FN uint32_t shf_r(uint32_t lo, uint32_t hi, uint32_t s) {  // low word of hi:lo >> (s % 32)
#if defined(__CUDA_ARCH__)
  return __funnelshift_r(lo, hi, s);
#else
  return static_cast<uint32_t>((static_cast<uint64_t>(hi) << 32 | lo) >> (s & 31u));
#endif
}

// Conversion of two binary64 values.  For x in [2^-7, 1) the exponent field is
// 1016 .. 1022 and the frame-59 integer is the significand shifted left by
// (field - 1016).  h comes from the leading 24 significand bits read as a
// binary32 (the word shifted left by three: the exponent field keeps its low
// eight bits, 248 .. 254, and its next bit lands in the sign, so the value is
// -x * 2^128), truncated to h's grid by adding and subtracting a base; m and l
// are cut out by funnel shifts whose amounts are taken modulo 32.
NPBGB_FX_FN uint32_t and_or(uint32_t a, uint32_t mask, uint32_t b) {  // (a & mask) | b
#if defined(__CUDA_ARCH__)
  uint32_t r;
  asm("lop3.b32 %0, %1, %2, %3, 0xea;" : "=r"(r) : "r"(a), "r"(mask), "r"(b));
  return r;
#else
  return (a & mask) | b;
#endif
}
struct Bits3 {
  uint32_t h, m, l;
};
NPBGB_FX_FN Bits3 cut(const Consts& k, uint32_t hi, uint32_t lo) {
  const uint32_t be = hi >> 20;
  const uint32_t mh = and_or(hi, 0xfffffu, k.implicit);
  return Bits3{shf_l(lo, hi, 3u), and_or(shf_l(lo, mh, be + 21u), 0xfffffu, first(k.m_base)),
               and_or(shf_l(0u, lo, be + 8u), 0x7ffffu, first(k.l_base))};
}
// Anything else: +0 is a value too, the rest is refused (NaN).
NPBGB_FX_FN Bits3 cut_other(uint32_t hi, uint32_t lo) {
  return Bits3{(hi | lo) == 0u ? 0u : kNaN, kMBase, kLBase};
}

NPBGB_FX_FN L3 from_f64(const Consts& k, uint64_t a, uint64_t b) {
  const uint32_t ah = static_cast<uint32_t>(a >> 32) - k.scale, al = static_cast<uint32_t>(a);
  const uint32_t bh = static_cast<uint32_t>(b >> 32) - k.scale, bl = static_cast<uint32_t>(b);
  Bits3 x = cut(k, ah, al), y = cut(k, bh, bl);
  // hi words of the range are 0x3f800000 .. 0x3fefffff
  const uint32_t ra = ah - 0x3f800000u, rb = bh - 0x3f800000u;
  if ((ra > rb ? ra : rb) >= 0x700000u) {
    if (ra >= 0x700000u) x = cut_other(ah + k.scale, al);
    if (rb >= 0x700000u) y = cut_other(bh + k.scale, bl);
  }
  return L3{fma(k.h_base, k.minus_one, fma_rz(pair(x.h, y.h), k.h_scale, k.h_base)),
            fma(k.m_base, k.minus_one, pair(x.m, y.m)), fma(k.l_base, k.minus_one, pair(x.l, y.l))};
}

// Consts::scale for values about as large as those sampled: `top` is the largest
// upper word of their finite non-negative ones.  Binary64 sums and products by
// constants commute with powers of two while nothing under- or overflows, so a frame
// may hold x * 2^-s.  Samples in [2^-4, 1) or none keep s = 0; otherwise the frame is
// [2^-7, 1) times a power of two of two to four times the largest sample.  |s| stays
// at most 100: then no other value's shifted word looks like one in range, and results
// stay far from both ends of binary64.
NPBGB_FX_FN uint32_t frame_of(uint32_t top) {
  const int e = static_cast<int>(top >> 20) - 1022;
  const bool keep = top == 0u || (e >= -3 && e <= 0) || e < -101 || e > 99;
  return keep ? 0u : static_cast<uint32_t>(e + 1) << 20;
}

// Whether from_f64 refuses the binary64 x.
NPBGB_FX_FN bool refused(const Consts& k, uint64_t x) {
  return static_cast<uint32_t>(x >> 32) - k.scale - 0x3f800000u >= 0x700000u && x != 0;
}
// Whether it refused either value.
NPBGB_FX_FN bool refused_value(const L3& x) {
  return (first(x.h) << 1) > 0xff000000u || (second(x.h) << 1) > 0xff000000u;
}
// Whether it refused both values.
NPBGB_FX_FN bool refused_both(const L3& x) {
  return (first(x.h) << 1) > 0xff000000u && (second(x.h) << 1) > 0xff000000u;
}

// T rounded in place; returns t's exponent fields, 2^e (in h's scale) of each
// sum as a binary32 pattern (0 for a zero sum, all ones for NaN).
NPBGB_FX_FN P2 round_pos(const Consts& k, L3& x, P2& t) {
  t = add_rz(x.h, fma_rz(x.l, k.l_to_m, x.m));
  const P2 e{t.v & kExpBoth};
  x.l = fma(e, k.minus_one, add(x.l, e));
  return e;
}
NPBGB_FX_FN P2 round_pos(const Consts& k, L3& x) {
  P2 t;
  return round_pos(k, x, t);
}
NPBGB_FX_FN P2 round_any(const Consts& k, L3& x) {
  const P2 t1 = add(x.h, x.m);
  const P2 err = add(x.m, fma(t1, k.minus_one, x.h));
  const P2 t = add_rz(t1, fma(x.l, k.l_to_m, err));
  const P2 e{t.v & kExpBoth};
  const P2 c = add(e, k.one);
  x.l = fma(c, k.minus_one, add(x.l, c));
  return e;
}

// e of one value is that of a sum in [2^lo, 2^hi) (NaN, zero and negative sums
// are not: the sign bit is cleared in e, so the caller's sums are known to be
// positive or zero).
template <int LO, int HI>
NPBGB_FX_FN bool within(uint32_t e) {
  return e - (static_cast<uint32_t>(135 + LO) << 23) < (static_cast<uint32_t>(HI - LO) << 23);
}

// A rounded sum of non-negative limbs, 2^-7 <= T < 8, read as T * 2^-(F - 59),
// in binary64: the limbs' patterns next to a base are integers, their weighted
// sum is T in units of 2^-59, and dropping the e + 7 low bits (zero after the
// rounding) leaves the significand; e's exponent field modulo 32 is e + 7.
struct Words {
  P2 h, m, l;
};
NPBGB_FX_FN Words words_of(const Consts& k, const L3& x) {
  return Words{add(x.h, k.h_base), add(x.m, k.m_base), add(x.l, k.l_base)};
}
// (h << 39) + (m << 19) + l, less the bases; the upper words' part of it.
constexpr uint64_t kBias = (static_cast<uint64_t>(kHBase) << 39) + (static_cast<uint64_t>(kMBase) << 19);
static_assert((kBias & 0xffffffffu) == 0, "the bases leave the low word alone");

// The sum as a frame-59 integer, for l >= 0.
NPBGB_FX_FN int64_t to_fx(uint32_t h, uint32_t m, uint32_t l) {
  const uint32_t top = h * 128u - static_cast<uint32_t>(kBias >> 32);
  return static_cast<int64_t>((static_cast<uint64_t>(top) << 32 | (l - kLBase)) +
                              static_cast<uint64_t>(m) * 0x80000u);
}

template <int F>
NPBGB_FX_FN uint64_t to_f64(uint32_t h, uint32_t m, uint32_t l, uint32_t e, uint32_t scale = 0) {
  const uint32_t top = h * 128u - static_cast<uint32_t>(kBias >> 32);
  // l may have been rounded to just below zero: its base comes off with a borrow
  const uint64_t x = (static_cast<uint64_t>(top) << 32 | l) + static_cast<uint64_t>(m) * 0x80000u - kLBase;
  const uint32_t xh = static_cast<uint32_t>(x >> 32), xl = static_cast<uint32_t>(x);
  const uint32_t s = e >> 23;
  const uint32_t lo = shf_r(xl, xh, s);
  const uint32_t hi = shf_r(xh, 0u, s) + (e >> 3) + (scale + (static_cast<uint32_t>(946 - F) << 20));
  return static_cast<uint64_t>(hi) << 32 | lo;
}

NPBGB_FX_FN P2 mul(P2 a, P2 b) {
#if defined(__CUDA_ARCH__)
  P2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
#else
  return each(a, b, b, [](float x, float y, float) { return x * y; });
#endif
}
// The larger magnitude of a and b below c (false if any of them is NaN).
NPBGB_FX_FN bool both_below(uint32_t a, uint32_t b, uint32_t c) {
#if defined(__CUDA_ARCH__)
  return fmaxf(fabsf(__uint_as_float(a)), fabsf(__uint_as_float(b))) < __uint_as_float(c);
#else
  const float x = std::fabs(f32_of(a)), y = std::fabs(f32_of(b));
  return (x > y || y != y ? x : y) < f32_of(c);
#endif
}

// RN(0.2 * s) of a rounded sum s of at most five values, with t as round_pos gave
// it, in limbs that are again non-negative and bounded (m < 2^-19, l < 2^-39: the
// limbs of five such values still add exactly).  `sure` says for each value whether
// the result stands; where it does not, it has to be evaluated another way.
//
// The double nearest 0.2 is (2^55 + 2) / (5 * 2^55), so the exact product is
// (s + s * 2^-54) / 5.  Long division of the limbs by five: h from t (so that no
// carry is left below), then m, each quotient truncated to its grid with a factor
// just below 1/5, each remainder exact; what is left is l1 = s - 5 (qh + qm), so
//   product = qh + qm + (l1 + s * 2^-54) / 5.
// The last term is rounded to a multiple u of the product's last place as in
// round_any (C = 1.5 * 2^e), from a binary32 estimate (whose error may exceed u/2
// for the smallest products); its remainder z = l1 - 5 ql + s * 2^-54, exact to
// 2^-20 u, corrects it, and what is then left of z decides: below 2.5 u (1 - 2^-18)
// in magnitude the rounding is IEEE's and not a tie.  e is the estimate's exponent,
// which stands unless the estimate lies within 2^-19 of a power of two: such
// products, ties, NaN, and products below 2^-7 are not sure.
NPBGB_FX_FN L3 fifth_of(const Consts& k, const L3& s, P2 t, bool& sure_a, bool& sure_b, P2& c) {
  L3 r;
  r.h = fma(k.h_base, k.minus_one, fma_rz(t, k.fifth, k.h_base));
  const P2 m1 = add(s.m, fma(k.minus_five, r.h, s.h));
  r.m = fma(k.m_base, k.minus_one, fma_rz(fma_rz(s.l, k.l_to_m, m1), k.fifth, k.m_base));
  const P2 l1 = fma(fma(k.minus_five, r.m, m1), k.m_to_l, s.l);
  const P2 y = mul(fma(t, k.t_to_l, l1), k.fifth);
  const P2 tr = add_rz(r.h, fma_rz(y, k.l_to_m, r.m));
  c = pair(and_or(first(tr), 0x7f800000u, k.half_bit), and_or(second(tr), 0x7f800000u, k.half_bit));
  const P2 q = fma(c, k.minus_one, add(y, c));
  const P2 z = fma(t, k.t_to_l, fma(k.minus_five, q, l1));
  const P2 d = fma(c, k.minus_one, fma(z, k.fifth, c));
  r.l = add(q, d);
  const P2 left = mul(fma(k.minus_five, d, z), k.z_scale);
  const P2 off = fma(c, k.minus_one, tr);
  const P2 limit = mul(c, k.third);
  sure_a = both_below(first(left), first(off), first(limit)) && first(c) >= 0x40400000u;
  sure_b = both_below(second(left), second(off), second(limit)) && second(c) >= 0x40400000u;
  return r;
}
NPBGB_FX_FN L3 fifth_of(const Consts& k, const L3& s, P2 t, bool& sure_a, bool& sure_b) {
  P2 c;
  return fifth_of(k, s, t, sure_a, sure_b, c);
}
// Its products in binary64, from the last argument's halves: their exponent fields
// with the bit below set, which to_f64 only sees in what it adds.
constexpr uint32_t kFifthScale = 0u - 0x80000u;

}  // namespace fxl
}  // namespace npbgb
