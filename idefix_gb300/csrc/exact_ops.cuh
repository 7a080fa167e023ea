// Exact FP64 operations formed from the bit patterns on the integer pipe.
//
// The FP64 pipe of this GPU is narrow and the FP64 kernels are bound by it
// while the integer pipe idles; where an FP64 operation has an exact result
// that the bit pattern gives directly, these helpers form it with integer
// operations.  Each equals the IEEE-754 operation it replaces for every
// input (NaNs compare false and stay NaN), checked on the host over random
// bit patterns, zeros, subnormals and infinities.
#pragma once
#include <stdint.h>

#include "fpconv.cuh"
#include "intdiv.cuh"  // dbits / dfrom, IDFX_HD

namespace idfx {

// Sign tests against zero from the bit pattern (FP64: integer pipe), equal
// to the IEEE comparisons for every x: zeros of either sign are neither > 0
// nor < 0, NaNs compare false.  FP32: the comparisons.
template <typename T>
IDFX_HD bool gt0(T x) {
  if constexpr (sizeof(T) == 8) {
    const int64_t b = (int64_t)dbits(x);
    return b > 0 && b <= 0x7FF0000000000000ll;
  } else {
    return x > T(0);
  }
}
template <typename T>
IDFX_HD bool lt0(T x) {
  if constexpr (sizeof(T) == 8) {
    const uint64_t m = dbits(x) & 0x7FFFFFFFFFFFFFFFull;  // |x|
    return (dbits(x) >> 63) && m != 0ull && m <= 0x7FF0000000000000ull;
  } else {
    return x < T(0);
  }
}
template <typename T>
IDFX_HD bool ge0(T x) {  // x >= 0: a zero or > 0
  if constexpr (sizeof(T) == 8) {
    return (dbits(x) << 1) == 0ull || gt0(x);
  } else {
    return x >= T(0);
  }
}
template <typename T>
IDFX_HD bool le0(T x) {
  if constexpr (sizeof(T) == 8) {
    return (dbits(x) << 1) == 0ull || lt0(x);
  } else {
    return x <= T(0);
  }
}

// x * s for a sign s = +-1 held as its sign bit (sb: 0 or the sign mask):
// on the FP64 path a sign-bit flip on the integer pipe, equal to the product
// for every non-NaN x; FP32 the product
template <typename T>
IDFX_HD T times_sign(T x, T s, uint64_t sb) {
  if constexpr (sizeof(T) == 8) {
    (void)s;
    return dfrom(dbits(x) ^ sb);
  } else {
    (void)sb;
    return x * s;
  }
}

// 0 x and x / 2
IDFX_HD double zero_times(double x) {  // (+0) x
  const uint64_t u = dbits(x);
  if (((u >> 52) & 0x7ffu) != 0x7ffu) return dfrom(u & (1ull << 63));
  return dfrom(0x7FF8000000000000ull);
}
IDFX_HD double half_of(double x) {
  const uint64_t u = dbits(x);
  const uint32_t e = (uint32_t)(u >> 52) & 0x7ffu;
  if (e - 2u < 2045u) return dfrom(u - (1ull << 52));
  if ((u << 1) == 0ull) return x;
  return rare_mul(0.5, x);
}

// x[A] .. x[B - 1] halved; false, and some of x left undefined, where one of
// them is neither zero nor far enough from the ends of the exponent range: one
// rare branch for all of them
template <int A, int B>
IDFX_HD bool halve(double* x) {
  bool ok = true;
#pragma unroll
  for (int n = A; n < B; n++) {
    const uint64_t u = dbits(x[n]);
    const uint32_t e = (uint32_t)(u >> 52) & 0x7ffu;
    ok = ok && (e - 64u < 1920u || (u << 1) == 0ull);
    x[n] = dfrom(e == 0u ? u : u - (1ull << 52));
  }
  return ok;
}

// x 2^K: on the FP64 path an add to the exponent field (the FP64 pipe is what
// the sweeps wait for), zeros as they are, and the product, as a call, where
// the result could leave the normal range; FP32 the product
template <int K, typename T>
IDFX_HD T pow2x(T x) {
  static_assert(K >= -1 && K <= 2, "half, twice, four times");
  constexpr double f = K < 0 ? 0.5 : (double)(1 << (K < 0 ? 0 : K));
  if constexpr (sizeof(T) == 8) {
    const uint64_t u = dbits(x);
    if (((uint32_t)(u >> 52) & 0x7ffu) - 64u < 1920u) return dfrom(u + ((uint64_t)(int64_t)K << 52));
    if ((u << 1) == 0ull) return x;
    return rare_mul(x, f);
  } else {
    return x * T(f);
  }
}

// x < y: on the FP64 path from the bit patterns (ordered as signed integers
// once the negative ones are reversed; zeros equal, NaNs false)
template <typename T>
IDFX_HD bool lt(T x, T y) {
  if constexpr (sizeof(T) == 8) {
    const uint64_t M = 0x7FFFFFFFFFFFFFFFull, I = 0x7FF0000000000000ull;
    const uint64_t u = dbits(x), w = dbits(y);
    if ((u & M) > I || (w & M) > I) return false;
    const int64_t a = (u >> 63) ? -(int64_t)(u & M) : (int64_t)u;
    const int64_t b = (w >> 63) ? -(int64_t)(w & M) : (int64_t)w;
    return a < b;
  } else {
    return x < y;
  }
}

// x <= y, and |x| >= |y|, the same way
template <typename T>
IDFX_HD bool le(T x, T y) {
  if constexpr (sizeof(T) == 8) {
    const uint64_t I = 0x7FF0000000000000ull << 1;
    return (dbits(x) << 1) <= I && (dbits(y) << 1) <= I && !lt(y, x);
  } else {
    return x <= y;
  }
}
template <typename T>
IDFX_HD bool abs_ge(T x, T y) {
  if constexpr (sizeof(T) == 8) {
    const uint64_t u = dbits(x) << 1, w = dbits(y) << 1, I = 0x7FF0000000000000ull << 1;
    return u <= I && w <= u;
  } else {
    return fabsf(x) >= fabsf(y);
  }
}

// neither infinite nor a NaN
template <typename T>
IDFX_HD bool is_finite(T x) {
  if constexpr (sizeof(T) == 8) {
    return (dbits(x) << 1) < (0x7FFull << 53);
  } else {
    return (fbits(x) << 1) < 0xFF000000u;
  }
}
template <typename T>
IDFX_HD T not_a_number() {
  if constexpr (sizeof(T) == 8) {
    return dfrom(0x7FF8000000000000ull);
  } else {
    return ffrom(0x7FC00000u);
  }
}

// the sign of x: -1, 0 (zeros, NaN) or 1; and s |x| for such a sign and
// x >= 0, the product's value (0 x where s is 0)
template <typename T>
IDFX_HD int sgn_of(T x) {
  return (int)gt0(x) - (int)lt0(x);
}
template <typename T>
IDFX_HD T times_sgn(int s, T x) {
  if constexpr (sizeof(T) == 8) {
    if (s == 0) return zero_times(x);
    return dfrom(dbits(x) ^ (s < 0 ? 1ull << 63 : 0ull));
  } else {
    return s * x;
  }
}

// x y < 0 and x y <= 0: on the FP64 path from the signs where both exponents
// are far enough from the ends for the product to be normal, else the product
template <typename T>
IDFX_HD bool prod_lt0(T x, T y) {
  if constexpr (sizeof(T) == 8) {
    const uint64_t u = dbits(x), w = dbits(y);
    if (((uint32_t)(u >> 52) & 0x7ffu) - 513u < 1022u && ((uint32_t)(w >> 52) & 0x7ffu) - 513u < 1022u)
      return ((u ^ w) >> 63) != 0ull;
    return lt0(rare_mul(x, y));
  } else {
    return x * y < T(0);
  }
}
template <typename T>
IDFX_HD bool prod_le0(T x, T y) {
  if constexpr (sizeof(T) == 8) {
    const uint64_t u = dbits(x), w = dbits(y);
    if (((uint32_t)(u >> 52) & 0x7ffu) - 513u < 1022u && ((uint32_t)(w >> 52) & 0x7ffu) - 513u < 1022u)
      return ((u ^ w) >> 63) != 0ull;
    return le0(rare_mul(x, y));
  } else {
    return x * y <= T(0);
  }
}

// x * s for a factor used many times: where s is a power of two (the face areas of
// boxes of 2^n cells a side) the product is an add to the exponent field on the
// FP64 path, with the product itself, as a call, outside the normal range
template <typename T>
struct Scale {
  T s;
  int k;  // s = 2^k, or the smallest int
};
template <typename T>
IDFX_HD Scale<T> scale_by(T s) {
  Scale<T> r{s, 0};
  if constexpr (sizeof(T) == 8) {
    const uint64_t u = dbits(s);
    const bool p = (u << 12) == 0ull && (u >> 52) - 1ull < 2046ull;  // positive, normal, a power of two
    r.k = p ? (int)(u >> 52) - 1023 : (int)0x80000000;
  }
  return r;
}
template <typename T>
IDFX_HD T scaled(T x, const Scale<T>& c) {
  if constexpr (sizeof(T) == 8) {
    if (c.k == (int)0x80000000) return x * c.s;
    const uint64_t u = dbits(x);
    const int e = (int)((uint32_t)(u >> 52) & 0x7ffu);
    if ((uint32_t)(e - 1) < 2046u && (uint32_t)(e + c.k - 1) < 2046u) return dfrom(u + ((uint64_t)(int64_t)c.k << 52));
    if ((u << 1) == 0ull) return x;
    return rare_mul(x, c.s);
  } else {
    return x * c.s;
  }
}

// One upwind term of CalcContactAverage, (1 - w) a + w b with the weight w
// in {0, 1/2, 1} (storeFlux.hpp:40-43).  The FP64 path forms the two
// products exactly on the integer pipe - a product by 1 is the value, by 0 a
// zero of the value's sign, by 1/2 an exponent decrement - and 1 - w from
// w's bit pattern, so only the sum issues on the FP64 pipe; any other weight,
// and non-finite or subnormal values, take the FP64 expression.  Every case
// is bit-identical to the reference's expression.
template <typename E>
IDFX_HD E upwind_term(E w, E a, E b) {
  if constexpr (sizeof(E) == 8) {
    const uint64_t W = dbits(w);
    double p, q;
    if (W == 0ull) {  // (1 - 0) a + 0 b
      p = a;
      q = zero_times(b);
    } else if (W == 0x3FF0000000000000ull) {  // (1 - 1) a + 1 b
      p = zero_times(a);
      q = b;
    } else if (W == 0x3FE0000000000000ull) {  // halves
      p = half_of(a);
      q = half_of(b);
    } else {
      p = rare_mul(rare_add(1.0, -w), a);
      q = rare_mul(w, b);
    }
    return p + q;
  } else {
    return (E(1) - w) * a + w * b;
  }
}

// upwind_term of the differences xa - ya and xb - yb.  FP64 path: for a weight
// of 0 or 1 (away from stagnant faces) the term is the picked difference, so
// only that one issues on the FP64 pipe - one operation instead of three; a
// zero difference (its sign would depend on the other's), a non-finite value on the
// other side (0 times it is NaN) and the weight 1/2 take the whole term, as a call.
IDFX_RARE double upwind_whole(double w, double xa, double ya, double xb, double yb) {
  return upwind_term(w, xa - ya, xb - yb);
}
template <typename E>
IDFX_HD E upwind_diff(E w, E xa, E ya, E xb, E yb) {
  if constexpr (sizeof(E) == 8) {
    const uint64_t W = dbits(w);
    const bool one = W == 0x3FF0000000000000ull;
    const double d = (one ? xb : xa) - (one ? yb : ya);
    const uint64_t ox = dbits(one ? xa : xb) << 1, oy = dbits(one ? ya : yb) << 1, F = 0x7FDull << 53;
    if ((one || W == 0ull) && ox < F && oy < F && (dbits(d) << 1) != 0ull) return d;
    return upwind_whole(w, xa, ya, xb, yb);
  } else {
    return upwind_term(w, xa - ya, xb - yb);
  }
}

// HLLD's degeneracy test, whether s1 - s < 1e-4 (sm - s) (left; right mirrored:
// s - s1 < 1e-4 (s - sm)).  FP64 path: a margin that FP32 arithmetic can see
// decides - each difference is within 2^-22 of the magnitudes of its FP64
// value, and where a magnitude is below FP32's normal range within 2^-148, which
// the smallest normal number in the margin covers - and the test itself, four
// FP64 operations a face, is a call.
IDFX_RARE bool degenerate_left(double s1, double s, double sm) { return lt(s1 - s, 1.e-4 * -(s - sm)); }
IDFX_RARE bool degenerate_right(double s1, double s, double sm) { return lt(-1.e-4 * (s - sm), s1 - s); }
template <bool LEFT, typename T>
IDFX_HD bool degenerate(T s1, T s, T sm) {
  if constexpr (sizeof(T) == 8) {
    const float a = d2f_rn(s1), b = d2f_rn(s), m = d2f_rn(sm);
    const float gap = LEFT ? a - b : b - a, all = LEFT ? m - b : b - m;
    if (gap - 1.e-4f * all > 9.5367431640625e-7f * (fabsf(a) + fabsf(b) + fabsf(m)) + 1.17549435e-38f) return false;
    return LEFT ? degenerate_left(s1, s, sm) : degenerate_right(s1, s, sm);
  } else {
    return LEFT ? lt(s1 - s, T(1.e-4) * -(s - sm)) : lt(T(-1.e-4) * (s - sm), s1 - s);
  }
}

// x / 4, the product's value
IDFX_HD float quarter(float x) { return 0.25f * x; }
IDFX_HD double quarter(double x) {
  const uint64_t u = dbits(x);
  if (((uint32_t)(u >> 52) & 0x7ffu) - 64u < 1920u) return dfrom(u - (2ull << 52));
  if ((u << 1) == 0ull) return x;
  return rare_mul(0.25, x);
}

}  // namespace idfx
