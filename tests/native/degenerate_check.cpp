// Host check of HLLD's degeneracy tests (exact_ops.cuh) against the FP64
// comparisons they stand for, with all three wave speeds of one magnitude
// drawn over the whole exponent range and, most of them, around the lower end
// of FP32's, where a conversion rounds by an absolute amount.  Prints the
// number of mismatches.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../idefix_gb300/csrc/exact_ops.cuh"

int main(int argc, char** argv) {
  const long n = argc > 1 ? std::atol(argv[1]) : 3000000;
  std::mt19937_64 rng(31);
  std::uniform_real_distribution<double> u(0.0, 1.0);
  unsigned long long mism = 0, total = 0;
  for (long i = 0; i < n; i++) {
    const int e = i % 4 ? -155 + (int)(rng() % 40) : -1060 + (int)(rng() % 2080);
    const double m = std::ldexp(1.0, e);
    const double s = (i % 3 ? -u(rng) : u(rng)) * m;
    const double d = (0.5 + u(rng)) * m * (i % 2 ? 1.0 : -1.0);  // sm - s
    // s1 at the threshold, a little to either side of it, or anywhere between
    const double f = i % 5 == 0 ? 1.e-4 : i % 5 < 4 ? 1.e-4 * (1.0 + 0.02 * (u(rng) - 0.5)) : u(rng);
    const double sm = s + d, s1 = s + d * f;
    const bool left = (s1 - s) < 1.e-4 * -(s - sm), right = -1.e-4 * (s - sm) < (s1 - s);
    total += 2;
    if (idfx::degenerate<true>(s1, s, sm) != left || idfx::degenerate<false>(s1, s, sm) != right) {
      if (mism < 10) std::printf("s1=%a s=%a sm=%a\n", s1, s, sm);
      mism++;
    }
  }
  std::printf("%llu mismatches of %llu\n", mism, total);
  return mism != 0;
}
