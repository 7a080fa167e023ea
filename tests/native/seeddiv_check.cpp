// Host check of idefix_gb300/csrc/seeddiv.cuh and the scalings and
// comparisons of exact_ops.cuh against IEEE-754: quotients and square roots
// over the whole exponent range and a moderate one, significands near 1 and 2
// and with few bits, equal and neighbouring operands, exact products and
// squares, special values.  Prints the number of mismatches.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../idefix_gb300/csrc/exact_ops.cuh"
#include "../../idefix_gb300/csrc/seeddiv.cuh"

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
  std::mt19937_64 rng(23);
  const uint64_t M = (1ull << 52) - 1;
  const double special[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 1e-310, -1e-310, 5e-324, 2.3e-308, 1.0, -1.0, 3.0,
                            1.7976931348623157e308};
  auto value = [&](int lo, int hi) {
    uint64_t m = rng() & M;
    switch (rng() % 5) {
      case 0: m &= ~((1ull << (rng() % 52)) - 1); break;  // few bits
      case 1: m = M - (rng() >> (12 + rng() % 50)); break;  // near 2
      case 2: m = rng() >> (12 + rng() % 50); break;        // near 1
    }
    return dfrom(((uint64_t)(lo + (long)(rng() % (uint64_t)(hi - lo + 1))) << 52) | m | (rng() & (1ull << 63)));
  };
  for (long i = 0; i < n; i++) {
    double a = i % 4 ? value(950, 1100) : value(0, 2047), b = i % 4 ? value(950, 1100) : value(0, 2047);
    switch (i % 16) {
      case 1: a = b; break;
      case 2: a = std::nextafter(b, a); break;
      case 3: a = b * (double)(1 + rng() % 64); break;
      case 4: a = special[rng() % (sizeof(special) / sizeof(special[0]))]; break;
      case 5: b = special[rng() % (sizeof(special) / sizeof(special[0]))]; break;
      case 6: a = b * value(950, 1100); break;
    }
    check("a / b", idfx::quot(a, b), a / b, a, b);
    double x = std::fabs(a);
    if (i % 8 == 1) x = b * b;
    if (i % 8 == 2) x = b * std::nextafter(b, 0.0);
    if (i % 64 == 7) x = a;
    check("sqrt", idfx::root(x), std::sqrt(x), x, 0.0);
    check("x / 2", idfx::pow2x<-1>(a), a * 0.5, a, 0.0);
    check("4 x", idfx::pow2x<2>(a), a * 4.0, a, 0.0);
    check("x < y", idfx::lt(a, b) ? 1.0 : 0.0, a < b ? 1.0 : 0.0, a, b);
  }
  std::printf("%llu mismatches in %llu checks\n", mism, total);
  return mism != 0;
}
