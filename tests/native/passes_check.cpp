// Host check of the helpers of the whole-array FP64 passes (exact_ops.cuh)
// against the IEEE-754 expressions they stand for: halved sums (RK2's
// combination, the mean of two faces), quarters, upwind terms whose side is
// picked before the difference, products by a power of two, and HLLD's
// degeneracy tests.  Prints the number of mismatches.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../idefix_gb300/csrc/exact_ops.cuh"

using idfx::dbits;
using idfx::dfrom;

static unsigned long long mism = 0, total = 0;

static void check(const char* what, double got, double want, double x, double y) {
  total++;
  if (dbits(got) != dbits(want) && !(std::isnan(got) && std::isnan(want))) {
    if (mism < 10) std::printf("%s mismatch x=%a y=%a: %a, not %a\n", what, x, y, got, want);
    mism++;
  }
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 3000000;
  std::mt19937_64 rng(29);
  const double special[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 5e-324, -5e-324, 1e-310, 2.3e-308, 1.0, -1.0,
                            1.7976931348623157e308, -1.7976931348623157e308};
  auto value = [&](int lo, int hi) {
    uint64_t m = rng() & ((1ull << 52) - 1);
    if (rng() % 3 == 0) m &= ~((1ull << (rng() % 52)) - 1);  // few bits: sums that tie or cancel
    return dfrom(((uint64_t)(lo + (long)(rng() % (uint64_t)(hi - lo + 1))) << 52) | m | (rng() & (1ull << 63)));
  };
  auto any = [&](long i) -> double {
    switch ((i + rng()) % 12) {
      case 0: return special[rng() % (sizeof(special) / sizeof(special[0]))];
      case 1: return value(0, 130);      // around the limit of the integer halving
      case 2: return value(1900, 2047);
      case 3: return value(0, 2047);
      default: return value(1000, 1040);
    }
  };
  long halved = 0;
  for (long i = 0; i < n; i++) {
    const double a = any(i), b = i % 16 == 3 ? -a : any(i + 1);
    double s[3] = {a + b, 7.0, a};
    if (idfx::halve<0, 1>(s)) {
      halved++;
      check("half sum", s[0], 0.5 * (a + b), a, b);
      check("sum of halves", s[0], 0.5 * a + 0.5 * b, a, b);
    }
    if (s[1] != 7.0) mism++;  // outside the range asked for
    double t[2] = {1.0, b};
    if (idfx::halve<0, 2>(t)) check("half", t[1], 0.5 * b, b, 0.0);
    check("quarter", idfx::quarter(a), 0.25 * a, a, 0.0);
    const double ya = i % 8 == 1 ? a : any(i + 2), xb = any(i + 3), yb = i % 8 == 2 ? xb : any(i + 4);
    const double w = i % 4 == 0 ? 0.0 : i % 4 == 1 ? 1.0 : i % 4 == 2 ? 0.5 : 0.3;
    const double sf = i % 3 ? std::ldexp(1.0, (int)(rng() % 140) - 120) : i % 9 ? value(1000, 1040) : any(i + 5);
    check("scaled", idfx::scaled(a, idfx::scale_by(sf)), a * sf, a, sf);
    // wave speeds: apart, nearly equal, at the threshold
    const double sl = i % 32 == 4 ? any(i) : value(1000, 1030), sm = i % 32 == 5 ? any(i + 1) : sl + value(1000, 1030);
    double s1 = i % 32 == 6 ? any(i + 2) : sl + (sm - sl) * (i % 2 ? 1e-4 : 1e-3 * (double)(rng() % 1000));
    for (uint64_t k = rng() % 4; k > 0; k--) s1 = std::nextafter(s1, i % 4 < 2 ? 1e300 : -1e300);
    if (i % 8 == 7) s1 += value(960, 1000);
    check("degenerate left", idfx::degenerate<true>(s1, sl, sm) ? 1 : 0, (s1 - sl) < 1.e-4 * -(sl - sm) ? 1 : 0, s1, sl);
    check("degenerate right", idfx::degenerate<false>(s1, sl, sm) ? 1 : 0, -1.e-4 * (sl - sm) < (s1 - sl) ? 1 : 0, s1, sl);
    check("upwind", idfx::upwind_diff(w, a, ya, xb, yb), (1.0 - w) * (a - ya) + w * (xb - yb), a, xb);
  }
  std::printf("%llu mismatches of %llu\n", mism, total);
  return mism != 0 || halved < n / 2;
}
