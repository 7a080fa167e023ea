// Correctly rounded FP64 quotients and square roots without the FP64 pipe.
//
// One FP64 instruction holds a scheduler's FP64 pipe for 64 cycles here (76
// with all four busy: about 520 G thread-operations per second for the whole
// GPU), while FP32 and integer instructions issue every cycle beside it; the
// flux sweeps run at that pipe's rate.  A hardware-sequence division takes
// 7.2 pipe operations, a square root 7.5, a reciprocal 4.5 (measured on
// independent chains).  Here a quotient is formed from the significands m
// and d (m in [d, 2 d)) with FP32 pairs and integers alone:
//   q0  m / d to about 41 bits in FP32 pairs - head and tail of both, a
//       hardware reciprocal f of d's head, one residual correction - as an
//       integer in units of 2^-42, two units low so that
//   r0 = m 2^42 - d q0      is positive (it fits 64 bits, so 64-bit wrapping
//                           arithmetic gives it exactly)
//   c  = the nearest integer to r0 2^10 f, twelve bits
//   r1 = r0 2^10 - d c      exact, within (1/2 + 2^-9) d of zero
// and q = q0 2^10 + c, one more or less where |r1| > d / 2 (equality cannot
// be: d has 53 bits and the quotient one bit more would have to divide it).
// The residual decides the rounding exactly, so the result is the IEEE one
// for every input, whatever the last bits of the seed.  The square root is the same
// with r0 = x 2^32 - s0^2 and r1 = r0 2^20 - c (s0 2^11 + c), against s: s is
// right exactly when -s < r1 <= s.  Exponents outside a safe band, zeros,
// subnormals, infinities and NaNs take the hardware operation.
// Measured on the 256^3 FP64 sweeps (x / y / z, both stages): hardware
// sequences 33.5 / 33.6 / 33.4 ms, a form with three FP64 operations per
// quotient (and the halves, fours and comparisons on the integer pipe) 27.5 /
// 27.1 / 26.6 ms with the marching sweep and 25.1 / 25.4 / 25.2 ms with a thread
// per cell, this form 19.1 / 19.4 / 19.2 ms.
// Newton's iteration with a residual test of the rounding, as in J.-M.
// Muller et al., Handbook of Floating-Point Arithmetic, ch. on division and
// square root.  Checked bit for bit against `/` and `sqrt` on the host and
// on the GPU.
#pragma once
#include <math.h>
#include <stdint.h>

#include "fpconv.cuh"  // fbits / ffrom
#include "intdiv.cuh"  // rcp_seed

namespace idfx {

// a called function on the device: some thirty quotients and roots of one
// face inlined are half of a sweep's instructions (256^3 sweeps 3 % slower)
#ifdef __CUDACC__
#define IDFX_CALL static __device__ __noinline__
#else
#define IDFX_CALL inline
#endif

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
IDFX_HD float clamp_f(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }

// exponent field inside [200, 1800)
IDFX_HD bool seed_band(uint32_t e) { return e - 200u < 1600u; }

// the significand of u with its leading one
IDFX_HD uint64_t significand(uint64_t u) { return (u & 0xfffffffffffffull) | (1ull << 52); }

// head and tail (24 + 23 bits) of the significand of u times 2^odd, in [1, 2)
// (odd = 0) or [2, 4)
IDFX_HD void seed_split(uint64_t u, uint32_t odd, float& h, float& l) {
  const uint32_t o = odd << 23;
  h = ffrom(((uint32_t)(u >> 29) & 0x7fffffu) + 0x3f800000u + o);
  l = ffrom((((uint32_t)u >> 6) & 0x7fffffu) + 0x34000000u + o) - ffrom(0x34000000u + o);
}

// head h in [1, 2) plus tail e f (|tail| < 2^-20) as an integer in units of
// 2^-42, `low` units less
IDFX_HD uint64_t seed_fixed(float h, float e, float f, uint32_t low) {
  const uint32_t m = 0x36400000u;  // 1.5 x 2^-19: its last place is 2^-42
  const int32_t t = (int32_t)(fbits(fma_f(e, f, ffrom(m))) - (m + low));
  return ((uint64_t)((fbits(h) & 0x7fffffu) | 0x800000u) << 19) + (uint64_t)(int64_t)t;
}

// nearest integer to x f 2^k, for 0 <= x f 2^k < 2^22
IDFX_HD uint32_t seed_round(uint32_t x, float f) {
  return fbits(fma_f((float)x, f, 8388608.0f)) - 0x4b000000u;
}

// a divisor prepared for several quotients
struct SeedDiv {
  double b;
  float h, l, f;  // significand head and tail, and the head's reciprocal
};

IDFX_HD SeedDiv seed_div(double b) {
  SeedDiv d;
  d.b = b;
  seed_split(dbits(b), 0u, d.h, d.l);
  d.f = rcp_seed(d.h);
  return d;
}

// a / D.b into q; false where the hardware division has to be taken
IDFX_HD bool try_quot(double a, const SeedDiv& D, double& q) {
  const uint64_t A = dbits(a), B = dbits(D.b);
  const uint32_t ea = (uint32_t)(A >> 52) & 0x7ffu;
  const uint32_t eb = (uint32_t)(B >> 52) & 0x7ffu;
  const uint64_t ma = significand(A), d = significand(B);
  const uint32_t up = ma < d ? 1u : 0u;  // m in [d, 2 d)
  const uint64_t m = ma << up;
  float ah, al;
  seed_split(A, up, ah, al);
  const float qh = clamp_f(ah * D.f, 1.0f, 1.99999988f);
  const float e = fma_f(-D.l, qh, fma_f(-D.h, qh, ah) + al);
  const uint64_t q0 = seed_fixed(qh, e, D.f, 2u);
  const uint64_t r0 = (m << 42) - d * q0;
  const uint32_t c = seed_round((uint32_t)(r0 >> 24), D.f * ffrom((127u - 18u) << 23));
  const int64_t r1 = (int64_t)((r0 << 10) - d * c);
  uint64_t z = (q0 << 10) + c;
  if (2 * r1 > (int64_t)d) z += 1ull;
  if (2 * r1 < -(int64_t)d) z -= 1ull;
  const uint32_t eq = ea - eb + 1022u - up;
  q = dfrom((z + ((uint64_t)eq << 52)) | ((A ^ B) & (1ull << 63)));
  return seed_band(ea) && seed_band(eb) && seed_band(eq);
}

// a / D.b, correctly rounded
IDFX_HD double quot(double a, const SeedDiv& D) {
  double q;
  if (try_quot(a, D, q)) return q;
  // zero dividends are common (states at rest, fields along an axis)
  const uint64_t A = dbits(a), B = dbits(D.b);
  if ((A << 1) == 0ull && seed_band((uint32_t)(B >> 52) & 0x7ffu)) return dfrom((A ^ B) & (1ull << 63));
  return rare_div(a, D.b);
}
// a / b, correctly rounded
IDFX_CALL double quot(double a, double b) { return quot(a, seed_div(b)); }

// sqrt(x), correctly rounded
IDFX_CALL double root(double x) {
  const uint64_t X = dbits(x);
  const uint32_t ex = (uint32_t)(X >> 52);  // with the sign bit: negative x is outside the band
  const uint32_t odd = (ex + 1u) & 1u;      // 2^(ex - 1023) = 2^odd 4^k
  const uint32_t k = (ex + 1u - odd) >> 1;  // k + 512
  const uint64_t m = significand(X) << odd;
  float h, l;
  seed_split(X, odd, h, l);
  const float f = rsqrt_seed(h);
  const float sh = clamp_f(h * f, 1.0f, 1.99999988f);
  const float e = fma_f(-sh, sh, h) + l;
  const uint64_t s0 = seed_fixed(sh, e, 0.5f * f, 2u);
  const uint64_t r0 = (m << 32) - s0 * s0;
  const uint32_t c = seed_round((uint32_t)(r0 >> 16), f * ffrom((127u - 17u) << 23));
  const int64_t r1 = (int64_t)((r0 << 20) - ((s0 << 11) + c) * c);
  uint64_t z = (s0 << 10) + c;
  if (r1 > (int64_t)z) {
    z += 1ull;
  } else if (r1 <= -(int64_t)z) {
    z -= 1ull;
  }
  if (seed_band(ex)) return dfrom(z + ((uint64_t)(k + 510u) << 52));
  return rare_sqrt(x);
}

}  // namespace idfx
