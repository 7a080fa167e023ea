// Correctly rounded FP64 quotients and square roots from FP32 seeds.
//
// One FP64 instruction holds a scheduler's FP64 pipe for 64 cycles here (76
// with all four busy: about 520 G thread-operations per second for the whole
// GPU), while FP32 and integer instructions issue every cycle beside it; the
// flux sweeps run at that pipe's rate.  A hardware-sequence division takes
// 7.2 pipe operations, a square root 7.5, a reciprocal 4.5 (measured on
// independent chains).  The forms below take three each:
//   q0   the quotient to about 42 bits, in FP32 pairs: the significands of
//        a and b as head + tail, a hardware reciprocal y of b's head, one
//        residual correction; assembled into a double with integer
//        operations
//   r0 = a - b q0            (one FMA)
//   q1 = q0 + r0 y           (one FMA; within 2^-11 ulp of a correctly
//                             rounded step: 42 + 22 bits)
//   r1 = a - b q1            (one FMA, exact)
// q1 is the correctly rounded quotient exactly when |r1| < |b| ulp(q1) / 2
// (half of that where q1 is a power of two, whose lower neighbour is nearer);
// the test compares the leading words of the bit patterns.  Where it does
// not hold (about one quotient in 2^11, and every quotient whose FP32 pair
// straddles a binade), or an exponent is outside a safe band, or an operand
// is zero, subnormal, infinite or NaN, the hardware operation gives the
// result.  So the result is the IEEE one for every input, whatever the
// accuracy of the seed.  The square root is the same with s1^2 in place of
// b q1: s1 is right exactly when |x - s1^2| < s1 ulp(s1) (x - s1^2 is a
// multiple of ulp(s1)^2, so the quarter-ulp^2 terms cannot matter).
// Measured with the limiter, HLLD and fast speeds on these forms (and the
// halves, fours and comparisons on the integer pipe): the three FP64 sweeps
// of 256^3 cells (PLM, HLLD, both stages) 33.5 / 33.6 / 33.4 -> 27.5 / 27.1 /
// 26.6 ms.
// Newton's iteration with a residual test of the rounding, as in J.-M.
// Muller et al., Handbook of Floating-Point Arithmetic, ch. on division and
// square root.  Checked bit for bit against `/` and `sqrt` on the host and
// on the GPU.
#pragma once
#include <math.h>
#include <stdint.h>

#include "fpconv.cuh"  // fbits / ffrom
#include "rdiv.cuh"    // fma_rn

namespace idfx {

// approximate 1 / sqrt of a float in [1, 4)
IDFX_HD float rsqrt_seed(float f) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  return r;
#else
  return 1.0f / sqrtf(f);
#endif
}
IDFX_HD float fma_f(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return fmaf(a, b, c);
#endif
}

// exponent field inside [200, 1800): products, residuals and ulps of such
// operands stay normal
IDFX_HD bool seed_band(uint32_t e) { return e - 200u < 1600u; }

// head and tail (24 + 23 bits) of the significand of u times 2^odd, in [1, 2)
// (odd = 0) or [2, 4)
IDFX_HD void seed_split(uint64_t u, uint32_t odd, float& h, float& l) {
  const uint32_t o = odd << 23;
  h = ffrom(((uint32_t)(u >> 29) & 0x7fffffu) + 0x3f800000u + o);
  l = ffrom((((uint32_t)u >> 6) & 0x7fffffu) + 0x34000000u + o) - ffrom(0x34000000u + o);
}

// the double head + tail (|tail| < 2^-20 of head's binade), times 2^(e - 896)
// and with the sign bit s: the tail rounded to 2^-42 of the binade
IDFX_HD double seed_join(float h, float l, uint32_t e, uint64_t s) {
  const uint32_t f = fbits(h);
  const uint32_t m = (f & 0x7f800000u) - (19u << 23) + 0x400000u;  // 1.5 x 2^-19 of the binade
  const int32_t t = (int32_t)(fbits(ffrom(m) + l) - m);
  return dfrom((((uint64_t)f << 29) + ((uint64_t)e << 52) + ((uint64_t)(int64_t)t << 10)) | s);
}

// the leading word of |x|
IDFX_HD uint32_t abs_hi(double x) { return (uint32_t)(dbits(x) >> 32) & 0x7fffffffu; }

// a divisor prepared for several quotients
struct SeedDiv {
  double b;
  double y;      // about 1 / b (22 bits)
  float h, l, f; // significand head and tail, and the head's reciprocal
  bool ok;       // b's exponent is inside the band
};

IDFX_HD SeedDiv seed_div(double b) {
  SeedDiv d;
  const uint64_t B = dbits(b);
  const uint32_t eb = (uint32_t)(B >> 52) & 0x7ffu;
  d.b = b;
  d.ok = seed_band(eb);
  seed_split(B, 0u, d.h, d.l);
  d.f = rcp_seed(d.h);
  d.y = dfrom((((uint64_t)fbits(d.f) << 29) + ((uint64_t)(1919u - eb) << 52)) ^ (B & (1ull << 63)));
  return d;
}

// a / d.b into q; false where the hardware division has to be taken
IDFX_HD bool try_seed_quot(double a, const SeedDiv& d, double& q) {
  const uint64_t A = dbits(a), B = dbits(d.b);
  const uint32_t ea = (uint32_t)(A >> 52) & 0x7ffu;
  const uint32_t eb = (uint32_t)(B >> 52) & 0x7ffu;
  float ah, al;
  seed_split(A, 0u, ah, al);
  const float qh = ah * d.f;
  const float e = fma_f(-d.l, qh, fma_f(-d.h, qh, ah) + al);
  const uint64_t s = (A ^ B) & (1ull << 63);
  const double q0 = seed_join(qh, e * d.f, 896u + ea - eb, s);
  const double r0 = fma_rn(-q0, d.b, a);
  const double q1 = fma_rn(r0, d.y, q0);
  const double r1 = fma_rn(-q1, d.b, a);
  const uint64_t Q = dbits(q1);
  // |b| ulp(q1) / 2: the exponents added, 1023 + 53 off; one less at a power of two
  uint32_t lim = abs_hi(d.b) + (((uint32_t)(Q >> 52) & 0x7ffu) << 20) - (1076u << 20);
  if ((Q << 12) == 0ull) lim -= 1u << 20;
  q = q1;
  return d.ok && seed_band(ea) && seed_band(ea - eb + 1023u) && abs_hi(r1) < lim;
}

// a / d.b, correctly rounded
IDFX_HD double quot(double a, const SeedDiv& d) {
  double q;
  if (try_seed_quot(a, d, q)) return q;
  return a / d.b;
}
// a / b, correctly rounded
IDFX_HD double quot(double a, double b) { return quot(a, seed_div(b)); }

// sqrt(x), correctly rounded
IDFX_HD double root(double x) {
  const uint64_t X = dbits(x);
  const uint32_t ex = (uint32_t)(X >> 52);  // with the sign bit: negative x is outside the band
  const uint32_t odd = (ex + 1u) & 1u;      // 2^(ex - 1023) = 2^odd 4^k
  const uint32_t k = (ex + 1u - odd) >> 1;  // k + 512
  float h, l;
  seed_split(X, odd, h, l);
  const float f = rsqrt_seed(h);
  const float sh = h * f;
  const float e = fma_f(-sh, sh, h) + l;
  const double s0 = seed_join(sh, e * (0.5f * f), 896u + k - 512u, 0ull);
  const double y = dfrom(((uint64_t)fbits(f) << 29) + ((uint64_t)(895u + 512u - k) << 52));  // about 1 / (2 sqrt(x))
  const double r0 = fma_rn(-s0, s0, x);
  const double s1 = fma_rn(r0, y, s0);
  const double r1 = fma_rn(-s1, s1, x);
  const uint64_t S = dbits(s1);
  // s1 ulp(s1): the exponents added, 1023 + 52 off; half at a power of two
  uint32_t lim = (uint32_t)(S >> 32) + (((uint32_t)(S >> 52) & 0x7ffu) << 20) - (1075u << 20);
  if ((S << 12) == 0ull) lim -= 1u << 20;
  if (seed_band(ex) && abs_hi(r1) < lim) return s1;
  return sqrt(x);
}

}  // namespace idfx
