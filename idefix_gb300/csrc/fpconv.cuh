// FP32 <-> FP64 conversions on the integer pipe.
//
// On this GPU the conversion instructions between FP32 and FP64 issue on the
// narrow FP64 pipe.  The mixed-precision path converts every primitive it
// hands to the FP32 sweeps and every FP32 EMF it hands to the FP64 face
// update; these two functions do it with integer operations on the bit
// patterns (IEEE-754 binary32 / binary64 layouts):
//   f2d_exact: binary32 -> binary64, exact (a rebias of the exponent and a
//              shift of the significand);
//   d2f_rn:    binary64 -> binary32, round to nearest, ties to even (half a
//              unit added before the 29 low significand bits are dropped; a
//              carry out of the significand moves into the exponent, up to
//              infinity as IEEE rounding does).
// Zeros take the integer path too; subnormal, infinite and NaN operands (and
// binary64 values outside the binary32 normal range) take the hardware
// conversion.  Both are checked bit for bit against the host's and CUDA's
// conversions.
#pragma once
#include <stdint.h>
#include <string.h>

#include "intdiv.cuh"  // dbits / dfrom, IDFX_HD

namespace idfx {

IDFX_HD uint32_t fbits(float x) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(x);
#else
  uint32_t u;
  memcpy(&u, &x, 4);
  return u;
#endif
}

IDFX_HD float ffrom(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  memcpy(&x, &u, 4);
  return x;
#endif
}

IDFX_HD double f2d_exact(float x) {
  const uint32_t u = fbits(x), t = u & 0x7fffffffu, s = u & 0x80000000u;
  if (t - 0x00800000u < 0x7f000000u) return dfrom(((uint64_t)(s | ((t >> 3) + (896u << 20))) << 32) | (u << 29));
  if (t == 0u) return dfrom((uint64_t)s << 32);
  return rare_widen(x);
}

IDFX_HD float d2f_rn(double x) {
  const uint64_t u = dbits(x);
  const uint32_t s = (uint32_t)(u >> 32) & 0x80000000u;
  // binary32 normal range: biased exponent 1..254 <=> binary64 897..1150
  if (((uint32_t)(u >> 52) & 0x7ffu) - 897u < 254u) {
    // half a unit of the last place kept, less one bit where that place is even
    const uint64_t r = u + ((1u << 28) - 1u + ((uint32_t)(u >> 29) & 1u));
    return ffrom(s | (((uint32_t)(r >> 29) - (896u << 23)) & 0x7fffffffu));
  }
  if ((u << 1) == 0ull) return ffrom(s);
  return rare_narrow(x);
}

}  // namespace idfx
