// Host check of npbench_gb300/csrc/divisor.cuh against the CPU's division.
//
// Built by tests/test_divisor.py with -ffp-contract=off.  Divisors and numerators
// are random, with runs of zeros and ones, and numerators are also placed next to
// divisor * (a number halfway between two binary64 values), where a quotient that
// is off by any amount rounds to the other side.  Prints "OK <count>" or the first
// mismatch.
#include <cinttypes>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../npbench_gb300/csrc/divisor.cuh"

using namespace npbgb;
using fx::bits_of;
using fx::double_of;

static std::mt19937_64 rng(99);

static double draw(uint64_t lo, uint64_t hi) {
  uint64_t m = rng() & ((1ull << 52) - 1);
  switch (rng() % 6) {
    case 0: m &= ~((1ull << (rng() % 52)) - 1); break;
    case 1: m |= (1ull << (rng() % 52)) - 1; break;
    case 2: m = rng() % 64; break;
    case 3: m = ((1ull << 52) - 1) - rng() % 64; break;
    default: break;
  }
  return double_of((lo + rng() % (hi - lo)) << 52 | m);
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
  auto check = [](double a, const Divisor& v) {
    const double want = a / v.d, got = div_by(a, v);
    if (bits_of(want) == bits_of(got) || (want != want && got != got)) return true;
    std::printf("MISMATCH %a / %a: want %a got %a\n", a, v.d, want, got);
    return false;
  };
  const double odd[] = {0.0, -0.0, 5e-324, -5e-324, 1e-300, 1e300, -1e308, INFINITY, -INFINITY, NAN};
  for (long i = 0; i < n; ++i) {
    const double d = i % 50 == 0 ? draw(1, 2046) * (i % 100 ? 1 : -1)
                   : i % 2       ? draw(1003, 1033)
                                 : 2.0 / double(1 + rng() % 4000) * (rng() % 2 ? 2.0 : 1.0);
    const Divisor v = divisor(d);
    if (!check(odd[rng() % 10], v)) return 1;
    double a = draw(900, 1100);
    if (rng() % 2) a = -a;
    if (!check(a, v)) return 1;
    if (!check(draw(1, 2046), v)) return 1;
    const double q = draw(950, 1050);                         // q + half a unit, times d
    const double half = double_of((bits_of(q) >> 52) << 52) * 0x1p-53;
    double near = std::fma(q, d, half * d);
    for (int s = -2; s <= 2; ++s)
      if (near > 0 && near < 1e300 && !check(double_of(bits_of(near) + uint64_t(int64_t(s))), v)) return 1;
  }
  std::printf("OK %ld\n", n);
  return 0;
}
