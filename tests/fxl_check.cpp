// Host check of npbench_gb300/csrc/fxl.cuh against the CPU's IEEE binary64.
//
// Built by tests/test_fxl.py with -ffp-contract=off.  For random and adversarial
// operands (ties, runs of zeros and ones, powers of two, nearly cancelling and
// equal neighbours, +0) it checks, bit for bit, conversion and the sums the
// kernels form: Heat-3D's update, Jacobi-2D's and Jacobi-1D's sums, and that
// values out of range are refused.  Prints "OK <count>" or the first mismatch.
#include <cinttypes>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../npbench_gb300/csrc/fxl.cuh"

using namespace npbgb;
using fx::bits_of;
using fx::double_of;

static std::mt19937_64 rng(4242);

static double draw() {
  const int kind = static_cast<int>(rng() % 9);
  if (kind == 0 && rng() % 4 == 0) return 0.0;
  const uint64_t e = 1016 + rng() % 7;
  uint64_t m = rng() & ((1ull << 52) - 1);
  if (kind == 1) m &= ~((1ull << (rng() % 52)) - 1);
  if (kind == 2) m |= (1ull << (rng() % 52)) - 1;
  if (kind == 3) m = 0;
  if (kind == 4) m = (1ull << 52) - 1;
  if (kind == 5) m &= (1ull << (1 + rng() % 20)) - 1;               // just above a power of two
  if (kind == 6) m = ((1ull << 52) - 1) ^ (rng() & ((1ull << (1 + rng() % 20)) - 1));
  return double_of(e << 52 | m);
}
// A value near x: a few units or a few low bits away, so that differences cancel.
static double near_to(double x) {
  double y = double_of(bits_of(x) + (rng() % 3 == 0 ? 0 : (rng() & ((1ull << (1 + rng() % 40)) - 1))) -
                       (rng() & ((1ull << (1 + rng() % 40)) - 1)));
  return (y >= 0.0078125 && y < 1.0) ? y : x;
}

static int fail(const char* what, const double* x, int n, uint64_t want, uint64_t got) {
  std::printf("MISMATCH %s: want %016" PRIx64 " got %016" PRIx64 ":", what, want, got);
  for (int i = 0; i < n; ++i) std::printf(" %a", x[i]);
  std::printf("\n");
  return 1;
}

static double heat(const double* x) {  // c, ip, im, jp, jm, kp, km
  volatile double c2 = 2.0 * x[0], d, t[3];
  for (int a = 0; a < 3; ++a) {
    d = x[1 + 2 * a] - c2;
    d = d + x[2 + 2 * a];
    t[a] = 0.125 * d;
  }
  d = t[0] + t[1];
  d = d + t[2];
  return d + x[0];
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 1000000;
  const fxl::Consts K = fxl::consts();
  long fifths = 0, unsure = 0, unsure_plain = 0, plain_sums = 0;
  long checks = 0, heats = 0, sums = 0;
  const double bad[] = {-0.0, 1.0, 0.0078124999999999, 5e-324, -0.5, 1e300, INFINITY, -INFINITY, NAN, 1e-300, 2.0};
  for (double b : bad) {
    const fxl::L3 r = fxl::from_f64(K, bits_of(b), bits_of(0.5));
    if ((fxl::first(r.h) & 0x7fffffffu) <= 0x7f800000u) return fail("refusal", &b, 1, 0, r.h.v);
    if ((fxl::second(r.h) & 0x7fffffffu) > 0x7f800000u) return fail("refusal of the other", &b, 1, 0, r.h.v);
  }
  for (long it = 0; it < n; ++it) {
    double x[7], y[7];
    const bool close = it % 3 == 0;
    for (int i = 0; i < 7; ++i) {
      x[i] = close && i ? near_to(x[0]) : draw();
      y[i] = draw();
    }
    // every tenth set is plain U[2^-7, 1): few of its products may be left open
    const bool kind_free = it % 10 == 9;
    if (kind_free) {
      for (int i = 0; i < 7; ++i) x[i] = 0.0078125 + (1.0 - 0.0078125) * double(rng() >> 11) * 0x1p-53;
      plain_sums += 5;
    }
    fxl::L3 v[7];
    for (int i = 0; i < 7; ++i) v[i] = fxl::from_f64(K, bits_of(x[i]), bits_of(y[i]));
    // Heat-3D
    {
      fxl::L3 s[3];
      for (int a = 0; a < 3; ++a) {
        s[a] = fxl::fma(K.minus_two, v[0], v[1 + 2 * a]);
        fxl::round_any(K, s[a]);
        s[a] = fxl::add(s[a], v[2 + 2 * a]);
        fxl::round_any(K, s[a]);
      }
      fxl::L3 w = fxl::add(s[0], s[1]);
      fxl::round_any(K, w);
      w = fxl::add(w, s[2]);
      fxl::round_any(K, w);
      w = fxl::fma(K.eight, v[0], w);
      const fxl::P2 e = fxl::round_any(K, w);
      const fxl::Words o = fxl::words_of(K, w);
      for (int half = 0; half < 2; ++half) {
        const double want = heat(half ? y : x);
        const uint32_t eh = half ? fxl::second(e) : fxl::first(e);
        if (!fxl::within<-4, 3>(eh)) {
          if (want >= 0.0078125 && want < 1.0) return fail("heat refused", half ? y : x, 7, bits_of(want), eh);
          continue;
        }
        const uint64_t got = half ? fxl::to_f64<62>(fxl::second(o.h), fxl::second(o.m), fxl::second(o.l), eh)
                                  : fxl::to_f64<62>(fxl::first(o.h), fxl::first(o.m), fxl::first(o.l), eh);
        if (got != bits_of(want)) return fail("heat", half ? y : x, 7, bits_of(want), got);
        ++heats;
      }
    }
    // the same values in a scaled frame: the same limbs, results scaled back; what no
    // frame holds stays refused
    {
      const int e = int(rng() % 201) - 100;
      fxl::Consts S = K;
      S.scale = static_cast<uint32_t>(e) << 20;
      fxl::L3 w{};
      for (int i = 0; i < 3; ++i) {
        w = fxl::from_f64(S, bits_of(std::ldexp(x[i], e)), bits_of(std::ldexp(y[i], e)));
        if (w.h.v != v[i].h.v || w.m.v != v[i].m.v || w.l.v != v[i].l.v)
          return fail("scaled frame", x + i, 1, v[i].h.v, w.h.v);
      }
      fxl::L3 sum = fxl::add(v[0], v[1]);
      const fxl::P2 se = fxl::round_pos(K, sum);
      const fxl::Words o = fxl::words_of(K, sum);
      if (fxl::within<-7, 3>(fxl::first(se))) {
        const uint64_t got =
            fxl::to_f64<59>(fxl::first(o.h), fxl::first(o.m), fxl::first(o.l), fxl::first(se), S.scale);
        if (got != bits_of(std::ldexp(x[0] + x[1], e))) return fail("scaled sum", x, 2, bits_of(x[0] + x[1]), got);
      }
      const double never[] = {-0.0, 5e-324, -0.5, INFINITY, -INFINITY, NAN, 1e-300, -std::ldexp(0.5, e), 1e300,
                              std::ldexp(1.0, e), std::ldexp(0.0078, e)};
      const double b = never[it % 11];
      const fxl::L3 r = fxl::from_f64(S, bits_of(b), bits_of(std::ldexp(0.5, e)));
      if ((fxl::first(r.h) & 0x7fffffffu) <= 0x7f800000u || (fxl::second(r.h) & 0x7fffffffu) > 0x7f800000u)
        return fail("scaled refusal", &b, 1, 0, r.h.v);
    }
    // sums of 3 and 5, in order
    fxl::L3 a = v[0];
    volatile double sx = x[0], sy = y[0];
    for (int i = 1; i < 5; ++i) {
      a = fxl::add(a, v[i]);
      const fxl::P2 e = fxl::round_pos(K, a);
      sx = sx + x[i];
      sy = sy + y[i];
      const fxl::Words o = fxl::words_of(K, a);
      if (fxl::within<-7, 3>(fxl::first(e))) {
        const uint64_t got = fxl::to_f64<59>(fxl::first(o.h), fxl::first(o.m), fxl::first(o.l), fxl::first(e));
        if (got != bits_of(sx)) return fail("sum", x, i + 1, bits_of(sx), got);
        ++sums;
      } else if (sx != 0.0) {
        return fail("sum refused", x, i + 1, bits_of(sx), 0);
      }
      if (fxl::within<-7, 3>(fxl::second(e))) {
        const uint64_t got = fxl::to_f64<59>(fxl::second(o.h), fxl::second(o.m), fxl::second(o.l), fxl::second(e));
        if (got != bits_of(sy)) return fail("sum", y, i + 1, bits_of(sy), got);
        ++sums;
      } else if (sy != 0.0) {
        return fail("sum refused", y, i + 1, bits_of(sy), 0);
      }
    }
    // 0.2 * (sum of five), repeated on its own results: the limbs it leaves are
    // inputs of the next round
    fxl::L3 z[5];
    double zx[5];
    for (int i = 0; i < 5; ++i) z[i] = v[i], zx[i] = x[i];
    for (int round = 0; round < 3; ++round) {
      fxl::L3 r[5];
      double rx[5];
      bool all = true;
      for (int j = 0; j < 5 && all; ++j) {
        fxl::L3 acc = z[j];
        volatile double sum = zx[j];
        fxl::P2 t{0};
        for (int i = 1; i < 5; ++i) {
          acc = fxl::add(acc, z[(j + i * (1 + round)) % 5]);
          sum = sum + zx[(j + i * (1 + round)) % 5];
          fxl::round_pos(K, acc, t);
        }
        bool sa, sb;
        r[j] = fxl::fifth_of(K, acc, t, sa, sb);
        rx[j] = 0.2 * sum;
        ++fifths;
        if (!sa) {
          ++unsure;
          all = false;
          if (sum != 0.0 && kind_free) ++unsure_plain;
          continue;
        }
        const fxl::Words o = fxl::words_of(K, r[j]);
        const double got = fx::to_f64<59>(fxl::to_fx(fxl::first(o.h), fxl::first(o.m), fxl::first(o.l)));
        if (bits_of(got) != bits_of(rx[j])) return fail("fifth", zx, 5, bits_of(rx[j]), bits_of(got));
      }
      if (!all) break;
      for (int i = 0; i < 5; ++i) z[i] = r[i], zx[i] = rx[i];
    }
    checks += 1;
  }
  if (plain_sums > 0 && unsure_plain * 2000 > plain_sums)
    return std::printf("MISMATCH too many products left open: %ld of %ld\n", unsure_plain, plain_sums), 1;
  if (heats < n || sums < 7 * n) return std::printf("MISMATCH too few values in range: %ld %ld\n", heats, sums), 1;
  std::printf("OK %ld (%ld of %ld products open, %ld of %ld on plain values)\n", checks, unsure, fifths,
              unsure_plain, plain_sums);
  return 0;
}
