// Device arithmetic of the ideal-MHD stage: cons/prim, physical flux, slope
// limiters, face reconstruction and the HLLD / HLL / Roe / TVDLF Riemann
// solvers, templated on the arithmetic type T.
//
// T = double is the parity path: compiled with --fmad=false, every
// expression keeps the operation order of the reference so that results are
// bit-identical to it (the reference's GPU CI also disables contraction,
// pytools/idfx_test.py:121).  Literals are written T(x), which is the same
// double for T = double.  T = float is the mixed-precision path (FP32
// reconstruction and Riemann solve; the callers keep the conserved state,
// cons->prim and the CT face update in FP64).
//
// D is the number of dimensions (= components, 2 or 3).  Variable order
// follows src/idefix.hpp:74-108: RHO, MX1..MXD, ENG(=PRS), BX1..BXD.
#pragma once
#include <cstdint>

#include "exact_ops.cuh"
#include "intdiv.cuh"
#include "seeddiv.cuh"

namespace idfx {

template <int D>
struct Var {
  static constexpr int NV = 2 * D + 2;
  static constexpr int RHO = 0, MX1 = 1, MX2 = 2, MX3 = 3;
  static constexpr int ENG = D + 1, PRS = D + 1;
  static constexpr int BX1 = D + 2, BX2 = D + 3, BX3 = D + 4;
};

// normal / tangent / bi-tangent indices for a sweep (hlldMHD.hpp:158-165)
template <int D, int DIR>
struct Dir {
  using V = Var<D>;
  static constexpr int Xn = V::MX1 + DIR;
  static constexpr int Xt = (DIR == 0 ? V::MX2 : V::MX1);
  static constexpr int Xb = (DIR == 2 ? V::MX2 : V::MX3);
  static constexpr int BXn = V::BX1 + DIR;
  static constexpr int BXt = (DIR == 0 ? V::BX2 : V::BX1);
  static constexpr int BXb = (DIR == 2 ? V::BX2 : V::BX3);
};

constexpr double kSmallPressureFix = 1.0e-5;  // fluid_defs.hpp:23
constexpr double kEpsUctContact = 1.0e-6;     // fluid_defs.hpp:24

// FP32 quotient for the mixed path: the approximate reciprocal (MUFU) and
// one FMA correction of the quotient, q' = q + (a - q b) r with q = a r
// (the correction step of Markstein's FMA division, P. W. Markstein, IBM J.
// Res. Dev. 34 (1990)): within about an ulp, at the cost of the bare
// reciprocal-multiply plus two FMAs; no special-case path (the mixed path
// divides by nonzero finite values; subnormals flush to zero).  Against IEEE
// division it leaves the mixed path's errors against FP64 unchanged while
// the bare reciprocal-multiply (2 ulp) had doubled them.
__device__ __forceinline__ float rcp_approx(float b) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(b));
  return r;
}
__device__ __forceinline__ float fdiv_corrected(float a, float b) {
  const float r = rcp_approx(b);
  const float q = a * r;
  const float e = __fmaf_rn(-q, b, a);
  return __fmaf_rn(e, r, q);
}

// division: FP64 IEEE correctly rounded (the bit-identical path; from FP32
// seeds and integers, off the FP64 pipe, seeddiv.cuh); FP32 (the mixed path,
// FP32-accurate rather than bit-matched) fdiv_corrected
template <typename T>
__device__ __forceinline__ T dv(T a, T b) {
  if constexpr (sizeof(T) == 4) {
    return fdiv_corrected(a, b);
  } else {
    return quot(a, b);
  }
}

// square root: FP64 IEEE (the bit-identical path, seeddiv.cuh); FP32 x * rsqrt(x), within
// 2 ulp (the tiny offset keeps sqrt(0) = 0; negative arguments stay NaN) -
// measured not to change the mixed path's errors against FP64
template <typename T>
__device__ __forceinline__ T sqr(T x) {
  if constexpr (sizeof(T) == 4) {
    return x * rsqrtf(x + 1.2e-38f);
  } else {
    return root(x);
  }
}

// 1 / b, as dv
template <typename T>
__device__ __forceinline__ T rcp(T b) {
  return dv(T(1), b);
}

// the quotient of the whole-array kernels (cons <-> prim) on the integer pipe
// for FP64 (intdiv.cuh): their quotients share a divisor, whose 64-bit
// reciprocal is formed once for all of them (the mixed stage end, when it took
// 1.96 ms per 256^3 cycle: 2.17 with the sweeps' quotients, 2.29 with calls of
// them)
template <typename T>
__device__ __forceinline__ T dvi(T a, T b) {
  if constexpr (sizeof(T) == 8) {
    return div_rn(a, b);
  } else {
    return a / b;
  }
}

// a b + c: one fused multiply-add on the FP32 (mixed) path; on the FP64
// path the product and the sum, rounded separately as the reference
// evaluates them (the library is built without FMA contraction), so that
// every FP64 expression written with it keeps the reference's bits
template <typename T>
__device__ __forceinline__ T mad(T a, T b, T c) {
  if constexpr (sizeof(T) == 4) {
    return fmaf(a, b, c);
  } else {
    return a * b + c;
  }
}

// sum of squares of the first D entries, in reference order
template <int D, typename T>
__device__ __forceinline__ T sumsq(T a, T b, T c) {
  T s = mad(b, b, a * a);
  if constexpr (D == 3) s = mad(c, c, s);
  return s;
}

// ---------------------------------------------------------------------------
// cons <-> prim (convertConsToPrim.hpp:15-100; eos_adiabatic.hpp:38-45)
// gm1 = gamma - 1.0, evaluated once on the host
// ---------------------------------------------------------------------------
// IPIPE: p / gm1 with the whole-array kernels' quotient (dvi), else with the
// sweeps' (dv); both correctly rounded.  bb = B^2 where the caller has it (HAVE_B2)
template <int D, bool IPIPE = false, bool HAVE_B2 = false, typename T>
__device__ __forceinline__ void prim_to_cons(T gm1, T* U, const T* V, T bb = T(0)) {
  using v = Var<D>;
  U[v::RHO] = V[v::RHO];
  U[v::MX1] = V[v::MX1] * V[v::RHO];
  U[v::MX2] = V[v::MX2] * V[v::RHO];
  if constexpr (D == 3) U[v::MX3] = V[v::MX3] * V[v::RHO];
  U[v::BX1] = V[v::BX1];
  U[v::BX2] = V[v::BX2];
  if constexpr (D == 3) U[v::BX3] = V[v::BX3];
  const T z = T(0);
  T kin, mag = bb;
  if constexpr (D == 3) {
    kin = sumsq<3>(V[v::MX1], V[v::MX2], V[v::MX3]);
    if constexpr (!HAVE_B2) mag = sumsq<3>(U[v::BX1], U[v::BX2], U[v::BX3]);
  } else {
    kin = sumsq<2>(V[v::MX1], V[v::MX2], z);
    if constexpr (!HAVE_B2) mag = sumsq<2>(U[v::BX1], U[v::BX2], z);
  }
  T pq;
  if constexpr (IPIPE) {
    pq = dvi(V[v::PRS], gm1);
  } else {
    pq = dv(V[v::PRS], gm1);
  }
  if constexpr (sizeof(T) == 8) {  // the halves exact on the integer pipe
    U[v::ENG] = pow2x<-1>(mag) + (pow2x<-1>(V[v::RHO]) * kin + pq);
  } else {
    U[v::ENG] = mad(T(0.5), mag, mad(T(0.5) * V[v::RHO], kin, pq));
  }
}

// FUSED (mixed path, FP64 state): the same FP64 pressure recovery with the
// sums of squares and the two subtractions as fused multiply-adds
// (p = (E - k m^2 - b^2 / 2) gm1 in 8 FP64 operations instead of 15, each
// fused step rounding once); the bit-exact path keeps the reference's
// operations
template <int D, bool INTDIV = false, typename T, bool FUSED = false>
__device__ __forceinline__ void cons_to_prim(T gm1, T* V, const T* U) {
  using v = Var<D>;
  auto q = [](T a, T b) { return INTDIV ? dvi(a, b) : dv(a, b); };
  if constexpr (FUSED) {
    V[v::RHO] = U[v::RHO];
    V[v::MX1] = q(U[v::MX1], U[v::RHO]);
    V[v::MX2] = q(U[v::MX2], U[v::RHO]);
    if constexpr (D == 3) V[v::MX3] = q(U[v::MX3], U[v::RHO]);
    V[v::BX1] = U[v::BX1];
    V[v::BX2] = U[v::BX2];
    if constexpr (D == 3) V[v::BX3] = U[v::BX3];
    T m2 = fma(U[v::MX2], U[v::MX2], U[v::MX1] * U[v::MX1]);
    T b2 = fma(U[v::BX2], U[v::BX2], U[v::BX1] * U[v::BX1]);
    if constexpr (D == 3) {
      m2 = fma(U[v::MX3], U[v::MX3], m2);
      b2 = fma(U[v::BX3], U[v::BX3], b2);
    }
    const T e = fma(-q(T(0.5), U[v::RHO]), m2, U[v::ENG]);
    V[v::PRS] = fma(T(-0.5), b2, e) * gm1;
    if (le0(V[v::PRS])) V[v::PRS] = T(kSmallPressureFix);
    return;
  }
  V[v::RHO] = U[v::RHO];
  V[v::MX1] = q(U[v::MX1], U[v::RHO]);
  V[v::MX2] = q(U[v::MX2], U[v::RHO]);
  if constexpr (D == 3) V[v::MX3] = q(U[v::MX3], U[v::RHO]);
  V[v::BX1] = U[v::BX1];
  V[v::BX2] = U[v::BX2];
  if constexpr (D == 3) V[v::BX3] = U[v::BX3];
  const T z = T(0);
  T m2, b2;
  if constexpr (D == 3) {
    m2 = sumsq<3>(U[v::MX1], U[v::MX2], U[v::MX3]);
    b2 = sumsq<3>(U[v::BX1], U[v::BX2], U[v::BX3]);
  } else {
    m2 = sumsq<2>(U[v::MX1], U[v::MX2], z);
    b2 = sumsq<2>(U[v::BX1], U[v::BX2], z);
  }
  const T kin = q(T(0.5), U[v::RHO]) * m2;
  const T mag = T(0.5) * b2;
  V[v::PRS] = (U[v::ENG] - kin - mag) * gm1;
  // floor; the reference's energy repair only touches a discarded local copy
  if (le0(V[v::PRS])) V[v::PRS] = T(kSmallPressureFix);
}

// induction flux of the transverse and bi-transverse field components
// (flux.hpp:28-95)
template <int D, int DIR, typename T>
__device__ __forceinline__ T flux_bt(const T* V) {
  using d = Dir<D, DIR>;
  return mad(V[d::Xn], V[d::BXt], -(V[d::BXn] * V[d::Xt]));
}
template <int D, int DIR, typename T>
__device__ __forceinline__ T flux_bb(const T* V) {
  using d = Dir<D, DIR>;
  return mad(V[d::Xn], V[d::BXb], -(V[d::BXn] * V[d::Xb]));
}

// physical MHD flux along DIR (flux.hpp:28-95); U is read before F is
// written; ptot = PRS + B^2 / 2 of the state where the caller has it
template <int D, int DIR, bool HAVE_PT = false, typename T>
__device__ __forceinline__ void phys_flux(T* F, const T* V, const T* U, T pt = T(0)) {
  using v = Var<D>;
  using d = Dir<D, DIR>;
  const T uXn = U[d::Xn], uE = U[v::ENG];
  const T u1 = U[v::MX1], u2 = U[v::MX2];
  T u3 = T(0);
  if constexpr (D == 3) u3 = U[v::MX3];
  F[v::RHO] = uXn;
  F[v::MX1] = mad(u1, V[d::Xn], -(V[d::BXn] * V[v::BX1]));
  F[v::MX2] = mad(u2, V[d::Xn], -(V[d::BXn] * V[v::BX2]));
  if constexpr (D == 3) F[v::MX3] = mad(u3, V[d::Xn], -(V[d::BXn] * V[v::BX3]));
  F[d::BXn] = T(0);
  F[d::BXt] = flux_bt<D, DIR>(V);
  if constexpr (D == 3) F[d::BXb] = flux_bb<D, DIR>(V);
  T vB;
  if constexpr (D == 3) {
    vB = mad(V[v::MX3], V[v::BX3], mad(V[v::MX2], V[v::BX2], V[v::MX1] * V[v::BX1]));
  } else {
    vB = mad(V[v::MX2], V[v::BX2], V[v::MX1] * V[v::BX1]);
  }
  T ptot = pt;
  if constexpr (!HAVE_PT) {
    T Bmag2;
    if constexpr (D == 3) {
      Bmag2 = sumsq<3>(V[v::BX1], V[v::BX2], V[v::BX3]);
    } else {
      Bmag2 = sumsq<2>(V[v::BX1], V[v::BX2], T(0));
    }
    if constexpr (sizeof(T) == 8) {
      ptot = pow2x<-1>(Bmag2) + V[v::PRS];
    } else {
      ptot = mad(T(0.5), Bmag2, V[v::PRS]);
    }
  }
  F[v::ENG] = mad(uE + ptot, V[d::Xn], -(V[d::BXn] * (vB)));
  F[d::Xn] += ptot;
}

// ---------------------------------------------------------------------------
// slope limiters (slopeLimiter.hpp)
// ---------------------------------------------------------------------------
// The reference MinModLim shadows its result variable and always returns 0
// (slopeLimiter.hpp:16-23); every "revert to minmod" path therefore adds 0.
template <typename T>
__device__ __forceinline__ T lim_minmod(T, T) {
  return T(0);
}

template <typename T>
__device__ __forceinline__ T lim_vanleer(T dvp, T dvm) {  // :54-57
  if (dvp * dvm > T(0)) return dv(T(2) * dvp * dvm, dvp + dvm);
  return T(0);
}

// half the van Leer slope on the FP64 path, 0.5 ((2 dvp) dvm) / (dvp + dvm):
// scaling by 2 is exact, so inside the seeded quotient's exponent band this
// is the correctly rounded (dvp dvm) / (dvp + dvm) - one product instead of
// three and no product by 1/2; outside it the expression as it stands
__device__ __forceinline__ double half_vanleer(double dvp, double dvm) {
  const double p = dvp * dvm;
  if (!gt0(p)) return 0.0;
  const double s = dvp + dvm;
  double q;
  if (try_quot(p, seed_div(s), q)) return q;
  return rare_mul(0.5, rare_div(rare_mul(rare_mul(2.0, dvp), dvm), s));
}

template <typename T>
__device__ __forceinline__ T lim_mc(T dvp, T dvm) {  // :68-76
  T dq = T(0);
  if (dvp * dvm > T(0)) {
    T dqc = T(0.5) * (dvp + dvm);
    T d2q = T(2) * (fabs(dvp) < fabs(dvm) ? dvp : dvm);
    dq = fabs(d2q) < fabs(dqc) ? d2q : dqc;
  }
  return dq;
}

// e2: (r dx)^2 and its correctly rounded reciprocal, formed on the host; the
// FP64 path divides by it and by 3 with Markstein's correction (rdiv.cuh),
// bit-identical to the divisions
template <typename T>
__device__ __forceinline__ T lim_limo3(T dvp, T dvm, T dx, double e2) {  // :25-52
  const T r = T(0.1), eps = T(1.e-12);
  T th = dv(dvm, dvp + T(1.e-16));
  T q;
  if constexpr (sizeof(T) == 8) {
    q = quot(T(2) + th, 3.0);
  } else {
    q = dv(T(2) + th, T(3));
  }
  T a = fmin(T(1.5), pow2x<1>(th));
  a = fmin(q, a);
  T b = fmax(-pow2x<-1>(th), a);
  T c = fmin(q, b);
  T psi = fmax(T(0), c);
  T eta = r * dx;
  if constexpr (sizeof(T) == 8) {
    eta = quot(dvm * dvm + dvp * dvp, e2);
  } else {
    (void)e2;
    eta = dv(dvm * dvm + dvp * dvp, eta * eta);
  }
  T lim;
  if (le(eta, T(T(1) - eps))) {
    lim = q;
  } else if (le(T(T(1) + eps), eta)) {
    lim = psi;
  } else {
    psi = (T(1) - dv(eta - T(1), eps)) * q + (T(1) + dv(eta - T(1), eps)) * psi;
    lim = T(0.5) * psi;
  }
  return lim;
}

// the limiter of a PPM face value vph between the cells v0 and vp1.  On the
// FP64 path the sign tests, the products by 1/2 and 2 and the signed minima
// are formed from the bit patterns: PPM is mostly such operations, and each
// would hold the FP64 pipe.
template <typename T>
__device__ __forceinline__ void ppm_limit_face(T vm1, T v0, T vp1, T vp2, T& vph) {  // :121-140
  if (prod_lt0(vp1 - vph, vph - v0)) {
    const T deltaL = (vm1 - pow2x<1>(v0) + vp1);
    const T deltaC = 3 * (v0 - pow2x<1>(vph) + vp1);
    const T deltaR = (v0 - pow2x<1>(vp1) + vp2);
    T delta = T(0);
    const int sc = sgn_of(deltaC);
    if (sgn_of(deltaL) == sc && sgn_of(deltaR) == sc) {
      const T C = T(1.25);
      delta = C * fmin(fabs(deltaL), fabs(deltaR));
      delta = times_sgn(sc, fmin(delta, fabs(deltaC)));
    }
    T d6;
    if constexpr (sizeof(T) == 8) {
      d6 = quot(delta, 6.0);
    } else {
      d6 = dv(delta, T(6));
    }
    vph = pow2x<-1>(v0 + vp1) - d6;
  }
}

// the limited PPM value of the face between the cells v0 and vp1: the left
// face value of one cell is the right face value of the cell before it
template <typename T>
__device__ __forceinline__ T ppm_face(T vm1, T v0, T vp1, T vp2) {
  const T c7 = T(7.0 / 12.0), c1 = T(1.0 / 12.0);
  T v = c7 * (v0 + vp1) - c1 * (vm1 + vp2);
  ppm_limit_face(vm1, v0, vp1, vp2, v);
  return v;
}
// second difference around v0
template <typename T>
__device__ __forceinline__ T ppm_diff2(T vm1, T v0, T vp1) {
  return vm1 + vp1 - pow2x<1>(v0);
}
// the cell's states from its limited face values vl, vr and the second
// differences around the cell before it, itself and the cell after it
template <typename T>
__device__ __forceinline__ void ppm_cell(T vm1, T v0, T vp1, T d2qcm1, T d2qc0, T d2qcp1, T& vl, T& vr) {  // :142-191
  T d2qf = T(6) * (vl + vr - pow2x<1>(v0));
  T d2q = T(0);
  const int sf = sgn_of(d2qf);
  if (sf == sgn_of(d2qc0) && sf == sgn_of(d2qcp1) && sf == sgn_of(d2qcm1)) {
    const T C = T(1.25);
    d2q = fmin(fabs(d2qc0), fabs(d2qcp1));
    d2q = C * fmin(fabs(d2qcm1), d2q);
    d2q = times_sgn(sf, fmin(fabs(d2qf), d2q));
  }
  T qmax = fmax(fmax(fabs(vm1), fabs(v0)), fabs(vp1));
  T rho = T(0);
  if (lt(T(1e-12) * qmax, fabs(d2qf))) rho = dv(d2q, d2qf);
  if (prod_le0(vr - v0, v0 - vl) || prod_le0(vm1 - v0, v0 - vp1)) {
    if (le(rho, T(T(1) - T(1e-12)))) {
      vl = v0 - rho * (v0 - vl);
      vr = v0 + rho * (vr - v0);
    }
  } else {
    if (abs_ge(vr - v0, pow2x<1>(v0 - vl))) vr = v0 + pow2x<1>(v0 - vl);
    if (abs_ge(vl - v0, pow2x<1>(v0 - vr))) vl = v0 + pow2x<1>(v0 - vr);
  }
}

template <typename T>
__device__ __forceinline__ void ppm_states(T vm2, T vm1, T v0, T vp1, T vp2, T& vl, T& vr) {
  vl = ppm_face(vm2, vm1, v0, vp1);
  vr = ppm_face(vm1, v0, vp1, vp2);
  ppm_cell(vm1, v0, vp1, ppm_diff2(vm2, vm1, v0), ppm_diff2(vm1, v0, vp1), ppm_diff2(v0, vp1, vp2), vl, vr);
}

// Cell-interface states of one cell from its stencil w[0..2*H] (centre w[H]):
// vl = value at its left face (the "vR" of that face), vr = value at its
// right face (the "vL" of the next face).  This is the per-cell form of
// ExtrapolateToFaces::ExtrapolatePrimVar (extrapolateToFaces.hpp:75-309):
// the reference evaluates the same limiter twice per cell (once for each
// face); here it is evaluated once and shared, with identical arithmetic.
// pos = true for RHO and PRS (positivity fallbacks of ORDER 3 and 4).
// ORDER 5 (learned) is the learned sweep's own (learned.cu); its stencil
// half-width is PLM's.
template <int ORDER>
struct Recon {
  static constexpr int H = (ORDER == 1 ? 0 : (ORDER == 4 ? 2 : 1));  // ORDER 5: 1
  // the positivity fall-back of the PPM states (van Leer slope)
  template <typename T>
  __device__ __forceinline__ static void ppm_positive(T vm1, T v0, T vp1, T& vl, T& vr) {
    if (le0(vr)) {
      T d = lim_vanleer(vp1 - v0, v0 - vm1);
      vr = v0 + T(0.5) * d;
    }
    if (le0(vl)) {
      T d = lim_vanleer(vp1 - v0, v0 - vm1);
      vl = v0 - T(0.5) * d;
    }
  }
  // PLM from the centre value and the differences on its two sides
  template <typename T>
  __device__ __forceinline__ static void plm(T w, T dvm, T dvp, bool shock, T& vl, T& vr) {
    if constexpr (sizeof(T) == 8) {
      const double h = shock ? 0.0 : half_vanleer(dvp, dvm);
      vr = w + h;
      vl = w - h;
    } else {
      const T d = shock ? lim_minmod(dvp, dvm) : lim_vanleer(dvp, dvm);
      vr = mad(T(0.5), d, w);
      vl = mad(T(-0.5), d, w);
    }
  }
  // shock: the cell is flagged by shock flattening (minmod slope, PLM and
  // LimO3 only, extrapolateToFaces.hpp:96-218)
  template <typename T>
  // e2: (0.1 dx)^2 (LimO3, FP64 path; Geo::l3b)
  __device__ __forceinline__ static void cell(const T* w, T dx, bool pos, T& vl, T& vr, bool shock = false,
                                              double e2 = 0.0) {
    if constexpr (ORDER == 1) {
      vl = w[0];
      vr = w[0];
    } else if constexpr (ORDER == 2) {
      const T dvm = w[1] - w[0];
      const T dvp = w[2] - w[1];
      plm(w[1], dvm, dvp, shock, vl, vr);
    } else if constexpr (ORDER == 3) {
      const T dm = w[1] - w[0];
      const T dp = w[2] - w[1];
      T d = shock ? lim_minmod(dp, dm) : dp * lim_limo3(dp, dm, dx, e2);
      vr = w[1] + pow2x<-1>(d);
      if (pos && le0(vr)) {
        d = lim_minmod(dp, dm);
        vr = w[1] + T(0.5) * d;
      }
      d = shock ? lim_minmod(dp, dm) : dm * lim_limo3(dm, dp, dx, e2);
      vl = w[1] - pow2x<-1>(d);
      if (pos && le0(vl)) {
        d = lim_minmod(dp, dm);
        vl = w[1] - T(0.5) * d;
      }
    } else {
      ppm_states(w[0], w[1], w[2], w[3], w[4], vl, vr);
      if (pos) ppm_positive(w[1], w[2], w[3], vl, vr);
    }
  }
};

// ---------------------------------------------------------------------------
// Riemann solvers.  In: face states vL, vR (BXn already set from Vs).
// Out: F, cmax, sl/sr (for uct_hll(d)), uL/uR (for uct_hlld).
// ---------------------------------------------------------------------------
enum Solver { kHLLD = 0, kHLL = 1, kROE = 2, kTVDLF = 3 };

template <int D, typename T>
struct RiemannOut {
  T F[Var<D>::NV];
  T uL[Var<D>::NV], uR[Var<D>::NV];
  T cmax, sl, sr;
};

// a / b where several quotients share b: on the FP64 path with the divisor
// prepared once (seeddiv.cuh); the FP32 path divides
template <typename T>
__device__ __forceinline__ T shared_div(T a, T b, const SeedDiv& R) {
  if constexpr (sizeof(T) == 8) {
    return quot(a, R);
  } else {
    return dv(a, b);
  }
}
template <typename T>
__device__ __forceinline__ SeedDiv shared_divisor(T b) {
  if constexpr (sizeof(T) == 8) {
    return seed_div(b);
  } else {
    return SeedDiv{};
  }
}

// fast magnetosonic speed of one face state (hlldMHD.hpp:205-238)
template <int D, int DIR, typename T>
__device__ __forceinline__ T fast_speed(T gamma, const T* v) {
  using vv = Var<D>;
  using d = Dir<D, DIR>;
  const T gpr = gamma * v[vv::PRS];
  const T b1 = v[d::BXn];
  const T b2 = v[d::BXt];
  T b3 = T(0);
  if constexpr (D == 3) b3 = v[d::BXb];
  const T Btmag2 = mad(b3, b3, b2 * b2);
  const T Bmag2 = mad(b1, b1, Btmag2);
  T c = gpr - Bmag2;
  if constexpr (sizeof(T) == 8) {  // products by 4 and 1/2 exact on the integer pipe
    c = gpr + Bmag2 + sqr(pow2x<2>(gpr) * Btmag2 + c * c);
    c = sqr(dv(pow2x<-1>(c), v[vv::RHO]));
  } else {
    c = gpr + Bmag2 + sqr(mad(T(4) * gpr, Btmag2, c * c));
    c = sqr(dv(T(0.5) * c, v[vv::RHO]));
  }
  return c;
}

template <int D, typename T>
__device__ __forceinline__ T b2_of(const T* v) {
  using vv = Var<D>;
  if constexpr (D == 3) return sumsq<3>(v[vv::BX1], v[vv::BX2], v[vv::BX3]);
  return sumsq<2>(v[vv::BX1], v[vv::BX2], T(0));
}
template <int D, typename T>
__device__ __forceinline__ T half_b2(const T* v) {
  return pow2x<-1>(b2_of<D>(v));
}

// HLLD (Miyoshi & Kusano 2005) with the reference's HLLC fall-back near
// degeneracy (hlldMHD.hpp:147-457, energy equation branch).
//
// The reference computes both sides' physical fluxes and star states and
// then picks one of five flux expressions (supersonic left / right, single
// star left / right, double star left / right).  Every one of them is the
// physical flux of ONE side plus corrections from that side's star states,
// so here the side is chosen first - from the same sign tests - and its
// operands are selected (integer selects of the bit patterns); the physical
// flux, the star momentum / energy and the double-star state are then
// evaluated for that side only, each with the reference's expression and
// operation order, so every face flux is bit-identical to the reference's.
// Only the HLLC fall-back reads the transverse-field fluxes of both sides.
// On the FP64 path this removes one physical flux, one side's star energy
// and momenta and one side's double-star state per face, and the divergent
// selection of the end (lanes of a warp on both sides issued both branches);
// the energy and the transverse momenta of the side not chosen are not formed
// either, and the degeneracy tests leave the FP64 pipe (with the flux times a
// face area that is a power of two: 309 -> 286 FP64 operations per cell and
// sweep, the 256^3 x / y / z sweeps of a cycle 19.1 / 19.3 / 19.2 -> 17.9 / 18.3 /
// 18.0 ms).
template <int D, int DIR, typename T>
__device__ __forceinline__ void riemann_hlld(T gamma, const T* vL, const T* vR, RiemannOut<D, T>& r) {
  using v = Var<D>;
  using d = Dir<D, DIR>;
  constexpr int NV = v::NV;
  constexpr int RHO = v::RHO, ENG = v::ENG, Xn = d::Xn, Xt = d::Xt, Xb = d::Xb;
  constexpr int BXn = d::BXn, BXt = d::BXt, BXb = d::BXb;
  T* uL = r.uL;
  T* uR = r.uR;
  const T cL = fast_speed<D, DIR>(gamma, vL);
  const T cR = fast_speed<D, DIR>(gamma, vR);
  const T cminL = vL[Xn] - cL, cmaxL = vL[Xn] + cL;
  const T cminR = vR[Xn] - cR, cmaxR = vR[Xn] + cR;
  const T sl = fmin(cminL, cminR);
  const T sr = fmax(cmaxL, cmaxR);
  r.sl = sl;
  r.sr = sr;
  r.cmax = fmax(fabs(sl), fabs(sr));
  const T gm1 = gamma - T(1);
  // of the conserved states both sides need the density, the normal momentum
  // and the field; the rest is formed for the chosen side below
  uL[RHO] = vL[RHO];
  uR[RHO] = vR[RHO];
  uL[Xn] = vL[Xn] * vL[RHO];
  uR[Xn] = vR[Xn] * vR[RHO];
#pragma unroll
  for (int n = v::BX1; n < NV; n++) {
    uL[n] = vL[n];
    uR[n] = vR[n];
  }
  const T bbL = b2_of<D>(vL), bbR = b2_of<D>(vR);
  const T ptL = vL[v::PRS] + pow2x<-1>(bbL);
  const T ptR = vR[v::PRS] + pow2x<-1>(bbR);
  // supersonic faces: the left physical flux if sl > 0, else the right one
  // if sr < 0; every other face is subsonic and takes star states
  bool sideL = gt0(sl);
  const bool sub = !(sideL || lt0(sr));
  bool dbl = false;
  T Bx = T(0), sBx = T(1), SM = T(0), pts = T(0), duL = T(0), duR = T(0);
  uint64_t sBxb = 0ull;
  T rhoL = T(0), rhoR = T(0), sqrL = T(0), sqrR = T(0), S1L = T(0), S1R = T(0);
  T dsL = T(0), dsR = T(0);
  T bn = T(0), bLt = T(0), bLb = T(0), bRt = T(0), bRb = T(0);  // star field components
  T vsL = T(0), vsR = T(0), wsL = T(0), wsR = T(0);
  if (sub) {
    T scrh = rcp(sr - sl);
    Bx = (sr * vR[BXn] - sl * vL[BXn]) * scrh;
    const bool bpos = gt0(Bx);
    sBx = (bpos ? T(1) : T(-1));
    sBxb = bpos ? 0ull : (1ull << 63);  // its sign bit
    duL = sl - vL[Xn];
    duR = sr - vR[Xn];
    scrh = rcp(duR * uR[RHO] - duL * uL[RHO]);
    SM = (duR * uR[Xn] - duL * uL[Xn] - ptR + ptL) * scrh;
    pts = duR * uR[RHO] * ptL - duL * uL[RHO] * ptR + vL[RHO] * vR[RHO] * duR * duL * (vR[Xn] - vL[Xn]);
    pts *= scrh;
    dsL = sl - SM;
    dsR = sr - SM;
    rhoL = dv(uL[RHO] * duL, dsL);
    rhoR = dv(uR[RHO] * duR, dsR);
    sqrL = sqr(rhoL);
    sqrR = sqr(rhoR);
    S1L = SM - dv(fabs(Bx), sqrL);
    S1R = SM + dv(fabs(Bx), sqrR);
    int revert_to_hllc = 0;
    if (degenerate<true>(S1L, sl, SM)) revert_to_hllc = 1;
    if (degenerate<false>(S1R, sr, SM)) revert_to_hllc = 1;
    if (revert_to_hllc) {
      // field components of the HLL state (sr uR - sl uL + FL - FR) / (sr - sl);
      // the normal component's fluxes are zero
      scrh = rcp(sr - sl);
      auto uhll = [&](T ul, T ur, T fl, T fr) {
        T u = sr * ur - sl * ul + fl - fr;
        u *= scrh;
        return u;
      };
      bn = uhll(uL[BXn], uR[BXn], T(0), T(0));
      bLt = bRt = uhll(uL[BXt], uR[BXt], flux_bt<D, DIR>(vL), flux_bt<D, DIR>(vR));
      if constexpr (D == 3) bLb = bRb = uhll(uL[BXb], uR[BXb], flux_bb<D, DIR>(vL), flux_bb<D, DIR>(vR));
      S1L = S1R = SM;
    } else {
      const T scrhL = dv(uL[RHO] * duL * duL - Bx * Bx, uL[RHO] * duL * dsL - Bx * Bx);
      const T scrhR = dv(uR[RHO] * duR * duR - Bx * Bx, uR[RHO] * duR * dsR - Bx * Bx);
      bn = Bx;
      bLt = uL[BXt] * scrhL;
      bRt = uR[BXt] * scrhR;
      if constexpr (D == 3) {
        bLb = uL[BXb] * scrhL;
        bRb = uR[BXb] * scrhR;
      }
    }
    const T scrhL = dv(Bx, uL[RHO] * duL);
    const T scrhR = dv(Bx, uR[RHO] * duR);
    vsL = vL[Xt] - scrhL * (bLt - uL[BXt]);
    vsR = vR[Xt] - scrhR * (bRt - uR[BXt]);
    if constexpr (D == 3) {
      wsL = vL[Xb] - scrhL * (bLb - uL[BXb]);
      wsR = vR[Xb] - scrhR * (bRb - uR[BXb]);
    }
    // single star left if S1L >= 0, else single star right if S1R <= 0,
    // else double star on the side of the contact (SM >= 0: left)
    sideL = ge0(S1L) || (!le0(S1R) && ge0(SM));
    dbl = !ge0(S1L) && !le0(S1R);
  }
  // the chosen side's primitive and conserved state (prim_to_cons with its
  // normal momentum and field from above) and its physical flux
  T vS[NV], uS[NV];
#pragma unroll
  for (int n = 0; n < NV; n++) vS[n] = sideL ? vL[n] : vR[n];
  prim_to_cons<D, false, true>(gm1, uS, vS, sideL ? bbL : bbR);
  uS[Xn] = sideL ? uL[Xn] : uR[Xn];
  T* F = r.F;
  const T pt = sideL ? ptL : ptR;
  phys_flux<D, DIR, true>(F, vS, uS, pt);  // pt: the same sum as the flux's total pressure
  if (!sub) return;
  // star state of the chosen side (us)
  const T s = sideL ? sl : sr;
  const T du = sideL ? duL : duR;
  const T vs = sideL ? vsL : vsR;
  const T ws = sideL ? wsL : wsR;
  T us[NV];
  us[RHO] = sideL ? rhoL : rhoR;
  us[BXn] = bn;
  us[BXt] = sideL ? bLt : bRt;
  if constexpr (D == 3) us[BXb] = sideL ? bLb : bRb;
  us[Xn] = us[RHO] * SM;
  us[Xt] = us[RHO] * vs;
  if constexpr (D == 3) us[Xb] = us[RHO] * ws;
  {
    T a = vS[Xn] * Bx + vS[Xt] * uS[BXt];
    if constexpr (D == 3) a = a + vS[Xb] * uS[BXb];
    T b = SM * Bx + vs * us[BXt];
    if constexpr (D == 3) b = b + ws * us[BXb];
    T scrh = a;
    scrh -= b;
    us[ENG] = du * uS[ENG] - pt * vS[Xn] + pts * SM + Bx * scrh;
    us[ENG] = dv(us[ENG], sideL ? dsL : dsR);
  }
  if (dbl) {
    // double-star state of the chosen side (uss); F += S1 (uss - us)
    const SeedDiv Rq = shared_divisor(sqrL + sqrR);  // divides the four double-star values
    T vss = sqrL * vsL + sqrR * vsR + times_sign(bRt - bLt, sBx, sBxb);
    vss = shared_div(vss, sqrL + sqrR, Rq);
    T wss = T(0);
    if constexpr (D == 3) {
      wss = sqrL * wsL + sqrR * wsR + times_sign(bRb - bLb, sBx, sBxb);
      wss = shared_div(wss, sqrL + sqrR, Rq);
    }
    T uss[NV];
    uss[RHO] = us[RHO];
    uss[Xn] = uss[RHO] * SM;
    uss[Xt] = uss[RHO] * vss;
    if constexpr (D == 3) uss[Xb] = uss[RHO] * wss;
    uss[BXn] = Bx;
    uss[BXt] = sqrL * bRt + sqrR * bLt + times_sign(sqrL * sqrR * (vsR - vsL), sBx, sBxb);
    uss[BXt] = shared_div(uss[BXt], sqrL + sqrR, Rq);
    if constexpr (D == 3) {
      uss[BXb] = sqrL * bRb + sqrR * bLb + times_sign(sqrL * sqrR * (wsR - wsL), sBx, sBxb);
      uss[BXb] = shared_div(uss[BXb], sqrL + sqrR, Rq);
    }
    T a = SM * Bx + vs * us[BXt];
    if constexpr (D == 3) a = a + ws * us[BXb];
    T b = SM * Bx + vss * uss[BXt];
    if constexpr (D == 3) b = b + wss * uss[BXb];
    T scrh = a;
    scrh -= b;
    // left: usL - sign(Bx) sqrL scrh, right: usR + sign(Bx) sqrR scrh; the
    // left difference is the sum with the sign-flipped term (IEEE defines
    // x - y as x + (-y), so the bits are the same)
    const T sq = sideL ? sqrL : sqrR;
    const T sgn = sideL ? -sBx : sBx;
    const uint64_t sgnb = sideL ? (sBxb ^ (1ull << 63)) : sBxb;
    uss[ENG] = us[ENG] + times_sign(sq * scrh, sgn, sgnb);
    const T S1 = sideL ? S1L : S1R;
    // density and normal momentum are the single star's: S1 times zero, which
    // is nothing or, where one of the two is not finite, a NaN (FP64: from the
    // bits, the two terms as they stand would be six FP64 operations a face)
    const bool fin = is_finite(S1);
#pragma unroll
    for (int n = 0; n < NV; n++) {
      if (sizeof(T) == 4 || (n != RHO && n != Xn)) F[n] = mad(S1, uss[n] - us[n], F[n]);
      else if (!(fin && is_finite(us[n]))) F[n] = not_a_number<T>();
    }
  }
  // F += s (us - u) of the chosen side: single star F = Fs + s (us - u),
  // double star F = (Fs + S1 (uss - us)) + s (us - u), the reference's order
#pragma unroll
  for (int n = 0; n < NV; n++) F[n] = mad(s, us[n] - uS[n], F[n]);
}

// HLL (hllMHD.hpp:154-453; the Hall whistler term is not part of ideal MHD)
template <int D, int DIR, typename T>
__device__ __forceinline__ void riemann_hll(T gamma, const T* vL, const T* vR, RiemannOut<D, T>& r) {
  using v = Var<D>;
  using d = Dir<D, DIR>;
  constexpr int NV = v::NV;
  T* uL = r.uL;
  T* uR = r.uR;
  T fluxL[NV], fluxR[NV];
  const T cL = fast_speed<D, DIR>(gamma, vL);
  const T cR = fast_speed<D, DIR>(gamma, vR);
  const T cminL = vL[d::Xn] - cL, cmaxL = vL[d::Xn] + cL;
  const T cminR = vR[d::Xn] - cR, cmaxR = vR[d::Xn] + cR;
  const T sl = fmin(cminL, cminR);
  const T sr = fmax(cmaxL, cmaxR);
  r.sl = sl;
  r.sr = sr;
  r.cmax = fmax(fabs(sl), fabs(sr));
  const T gm1 = gamma - T(1);
  prim_to_cons<D>(gm1, uL, vL);
  prim_to_cons<D>(gm1, uR, vR);
  phys_flux<D, DIR>(fluxL, vL, uL);
  phys_flux<D, DIR>(fluxR, vR, uR);
  T* F = r.F;
  if (sl > T(0)) {
#pragma unroll
    for (int n = 0; n <= D; n++) F[n] = fluxL[n];
  } else if (sr < T(0)) {
#pragma unroll
    for (int n = 0; n <= D; n++) F[n] = fluxR[n];
  } else {
#pragma unroll
    for (int n = 0; n <= D; n++)
      F[n] = dv(sl * sr * uR[n] - sl * sr * uL[n] + sr * fluxL[n] - sl * fluxR[n], sr - sl);
  }
  if (sl > T(0)) {
#pragma unroll
    for (int n = v::BX1; n < v::BX1 + D; n++) F[n] = fluxL[n];
    F[v::ENG] = fluxL[v::ENG];
  } else if (sr < T(0)) {
#pragma unroll
    for (int n = v::BX1; n < v::BX1 + D; n++) F[n] = fluxR[n];
    F[v::ENG] = fluxR[v::ENG];
  } else {
#pragma unroll
    for (int n = v::BX1; n < v::BX1 + D; n++) {
      F[n] = sl * sr * uR[n] - sl * sr * uL[n] + sr * fluxL[n] - sl * fluxR[n];
      F[n] *= rcp(sr - sl);
    }
    F[v::ENG] = sl * sr * uR[v::ENG] - sl * sr * uL[v::ENG] + sr * fluxL[v::ENG] - sl * fluxR[v::ENG];
    F[v::ENG] *= rcp(sr - sl);
  }
}

// TVDLF / Rusanov (tvdlfMHD.hpp:140-232)
template <int D, int DIR, typename T>
__device__ __forceinline__ void riemann_tvdlf(T gamma, const T* vL, const T* vR, RiemannOut<D, T>& r) {
  using v = Var<D>;
  using d = Dir<D, DIR>;
  constexpr int NV = v::NV;
  T vv[NV];
#pragma unroll
  for (int n = 0; n < NV; n++) vv[n] = T(0.5) * (vL[n] + vR[n]);
  const T gpr = gamma * vv[v::PRS];
  T Bt2 = T(0) + vv[d::BXt] * vv[d::BXt];
  if constexpr (D == 3) Bt2 = Bt2 + vv[d::BXb] * vv[d::BXb];
  const T B2 = Bt2 + vv[d::BXn] * vv[d::BXn];
  T cRL = gpr - B2;
  cRL = cRL + B2 + sqr(cRL * cRL + T(4) * gpr * Bt2);
  cRL = sqr(dv(T(0.5) * cRL, vv[v::RHO]));
  const T cmax = fmax(fabs(vv[d::Xn] + cRL), fabs(vv[d::Xn] - cRL));
  r.sl = -cmax;
  r.sr = cmax;
  r.cmax = cmax;
  T fluxL[NV], fluxR[NV];
  const T gm1 = gamma - T(1);
  prim_to_cons<D>(gm1, r.uL, vL);
  prim_to_cons<D>(gm1, r.uR, vR);
  phys_flux<D, DIR>(fluxL, vL, r.uL);
  phys_flux<D, DIR>(fluxR, vR, r.uR);
#pragma unroll
  for (int n = 0; n < NV; n++) r.F[n] = T(0.5) * (fluxL[n] + fluxR[n] + cmax * (r.uL[n] - r.uR[n]));
}

// Roe with the entropy fix (roeMHD.hpp:175-650, energy equation branch)
template <int D, int DIR, typename T>
__device__ __forceinline__ void riemann_roe(T gamma, const T* vL, const T* vR, RiemannOut<D, T>& r) {
  using v = Var<D>;
  using d = Dir<D, DIR>;
  constexpr int NV = v::NV;
  constexpr int RHO = v::RHO, ENG = v::ENG, PRS = v::PRS, Xn = d::Xn, Xt = d::Xt, Xb = d::Xb;
  constexpr int BXn = d::BXn, BXt = d::BXt, BXb = d::BXb;
  constexpr int KFASTM = 0, KFASTP = 1, KDIVB = 2, KENTRP = 3, KSLOWM = 4, KSLOWP = 5, KALFVM = 6,
                KALFVP = 7;
  const T delta = T(1.e-6);
  T dV[NV], dU[NV], fluxL[NV], fluxR[NV];
  T Rc[NV][NV];
  T* uL = r.uL;
  T* uR = r.uR;
#pragma unroll
  for (int n = 0; n < NV; n++) dV[n] = vR[n] - vL[n];
  const T gm1 = gamma - T(1);
  prim_to_cons<D>(gm1, uL, vL);
  prim_to_cons<D>(gm1, uR, vR);
#pragma unroll
  for (int n = 0; n < NV; n++) dU[n] = uR[n] - uL[n];
  phys_flux<D, DIR>(fluxL, vL, uL);
  phys_flux<D, DIR>(fluxR, vR, uR);
#pragma unroll
  for (int a = 0; a < NV; a++)
#pragma unroll
    for (int b = 0; b < NV; b++) Rc[a][b] = T(0);
  const T sqr_rho_L = sqr(vL[RHO]);
  const T sqr_rho_R = sqr(vR[RHO]);
  const T sl = dv(sqr_rho_L, sqr_rho_L + sqr_rho_R);
  const T sr = dv(sqr_rho_R, sqr_rho_L + sqr_rho_R);
  const T rho = sr * vL[RHO] + sl * vR[RHO];
  const T sqrt_rho = sqr(rho);
  T w = T(0), Bz = T(0), bz = T(0);
  const T u = sl * vL[Xn] + sr * vR[Xn];
  const T vv = sl * vL[Xt] + sr * vR[Xt];
  if constexpr (D == 3) w = sl * vL[Xb] + sr * vR[Xb];
  const T Bx = sr * vL[BXn] + sl * vR[BXn];
  const T By = sr * vL[BXt] + sl * vR[BXt];
  if constexpr (D == 3) Bz = sr * vL[BXb] + sl * vR[BXb];
  const T sBx = (Bx >= T(0) ? T(1) : T(-1));
  const T bx = dv(Bx, sqrt_rho);
  const T by = dv(By, sqrt_rho);
  if constexpr (D == 3) bz = dv(Bz, sqrt_rho);
  T bt2 = T(0) + by * by;
  if constexpr (D == 3) bt2 = bt2 + bz * bz;
  const T b2 = bx * bx + bt2;
  const T Btmag = sqr(bt2 * rho);
  T X = dV[BXn] * dV[BXn] + dV[BXt] * dV[BXt];
  if constexpr (D == 3) X = X + dV[BXb] * dV[BXb];
  X = dv(X, (sqr_rho_L + sqr_rho_R) * (sqr_rho_L + sqr_rho_R) * T(2));
  T Bmag2L, Bmag2R, vdm, BdB, vel2;
  if constexpr (D == 3) {
    Bmag2L = sumsq<3>(vL[v::BX1], vL[v::BX2], vL[v::BX3]);
    Bmag2R = sumsq<3>(vR[v::BX1], vR[v::BX2], vR[v::BX3]);
    vdm = u * dU[Xn] + vv * dU[Xt] + w * dU[Xb];
    BdB = Bx * dU[BXn] + By * dU[BXt] + Bz * dU[BXb];
    vel2 = u * u + vv * vv + w * w;
  } else {
    Bmag2L = sumsq<2>(vL[v::BX1], vL[v::BX2], T(0));
    Bmag2R = sumsq<2>(vR[v::BX1], vR[v::BX2], T(0));
    vdm = u * dU[Xn] + vv * dU[Xt];
    BdB = Bx * dU[BXn] + By * dU[BXt];
    vel2 = u * u + vv * vv;
  }
  const T pL = vL[PRS] + T(0.5) * Bmag2L;
  const T pR = vR[PRS] + T(0.5) * Bmag2R;
  dV[PRS] = (gamma - T(1)) * ((T(0.5) * vel2 - X) * dV[RHO] - vdm + dU[ENG] - BdB);
  const T HL = dv(uL[ENG] + pL, vL[RHO]);
  const T HR = dv(uR[ENG] + pR, vR[RHO]);
  const T H = sl * HL + sr * HR;
  const T Hgas = H - b2;
  const T a2 = (T(2) - gamma) * X + (gamma - T(1)) * (Hgas - T(0.5) * vel2);
  T scrh = a2 - b2;
  const T ca2 = bx * bx;
  scrh = scrh * scrh + T(4) * bt2 * a2;
  scrh = sqr(scrh);
  const T cf2 = T(0.5) * (a2 + b2 + scrh);
  const T cs2 = dv(a2 * ca2, cf2);
  const T cf = sqr(cf2);
  const T cs = sqr(cs2);
  const T ca = sqr(ca2);
  const T a = sqr(a2);
  T alpha_f, alpha_s;
  if (cf == cs) {
    alpha_f = T(1);
    alpha_s = T(0);
  } else if (a <= cs) {
    alpha_f = T(0);
    alpha_s = T(1);
  } else if (cf <= a) {
    alpha_f = T(1);
    alpha_s = T(0);
  } else {
    scrh = rcp(cf2 - cs2);
    alpha_f = (a2 - cs2) * scrh;
    alpha_s = (cf2 - a2) * scrh;
    alpha_f = fmax(T(0), alpha_f);
    alpha_s = fmax(T(0), alpha_s);
    alpha_f = sqr(alpha_f);
    alpha_s = sqr(alpha_s);
  }
  T beta_y, beta_z = T(0);
  if constexpr (D == 2) {
    beta_y = (Btmag > T(1.e-9)) ? ((By) >= T(0) ? T(1) : T(-1)) : T(1);
  } else {
    if (Btmag > T(1.e-9)) {
      beta_y = dv(By, Btmag);
      beta_z = dv(Bz, Btmag);
    } else {
      beta_z = beta_y = T(1);
    }
  }
  T lambda[NV], alambda[NV], eta[NV];
  T beta_dv = T(0) + beta_y * dV[Xt];
  T beta_dB = T(0) + beta_y * dV[BXt];
  T beta_v = T(0) + beta_y * vv;
  if constexpr (D == 3) {
    beta_dv = beta_dv + beta_z * dV[Xb];
    beta_dB = beta_dB + beta_z * dV[BXb];
    beta_v = beta_v + beta_z * w;
  }
  const T half_a2 = dv(T(0.5), a2);
  int kk = KFASTM;
  lambda[kk] = u - cf;
  scrh = alpha_s * cs * sBx;
  Rc[RHO][kk] = alpha_f;
  Rc[Xn][kk] = alpha_f * lambda[kk];
  Rc[Xt][kk] = alpha_f * vv + scrh * beta_y;
  if constexpr (D == 3) Rc[Xb][kk] = alpha_f * w + scrh * beta_z;
  Rc[BXt][kk] = dv(alpha_s * a * beta_y, sqrt_rho);
  if constexpr (D == 3) Rc[BXb][kk] = dv(alpha_s * a * beta_z, sqrt_rho);
  Rc[ENG][kk] = alpha_f * (Hgas - u * cf) + scrh * beta_v + dv(alpha_s * a * Btmag, sqrt_rho);
  eta[kk] = alpha_f * (X * dV[RHO] + dV[PRS]);
  eta[kk] += rho * scrh * beta_dv - rho * alpha_f * cf * dV[Xn] + sqrt_rho * alpha_s * a * beta_dB;
  eta[kk] *= half_a2;

  kk = KFASTP;
  lambda[kk] = u + cf;
  Rc[RHO][kk] = alpha_f;
  Rc[Xn][kk] = alpha_f * lambda[kk];
  Rc[Xt][kk] = alpha_f * vv - scrh * beta_y;
  if constexpr (D == 3) Rc[Xb][kk] = alpha_f * w - scrh * beta_z;
  Rc[BXt][kk] = Rc[BXt][KFASTM];
  if constexpr (D == 3) Rc[BXb][kk] = Rc[BXb][KFASTM];
  Rc[ENG][kk] = alpha_f * (Hgas + u * cf) - scrh * beta_v + dv(alpha_s * a * Btmag, sqrt_rho);
  eta[kk] = alpha_f * (X * dV[RHO] + dV[PRS]) - rho * scrh * beta_dv + rho * alpha_f * cf * dV[Xn] +
            sqrt_rho * alpha_s * a * beta_dB;
  eta[kk] *= half_a2;

  kk = KENTRP;
  lambda[kk] = u;
  Rc[RHO][kk] = T(1);
  Rc[Xn][kk] = u;
  Rc[Xt][kk] = vv;
  if constexpr (D == 3) Rc[Xb][kk] = w;
  Rc[ENG][kk] = T(0.5) * vel2 + dv(gamma - T(2), gamma - T(1)) * X;
  eta[kk] = dv((a2 - X) * dV[RHO] - dV[PRS], a2);

  kk = KDIVB;
  lambda[kk] = u;
  eta[kk] = T(0);

  scrh = alpha_f * cf * sBx;
  kk = KSLOWM;
  lambda[kk] = u - cs;
  Rc[RHO][kk] = alpha_s;
  Rc[Xn][kk] = alpha_s * lambda[kk];
  Rc[Xt][kk] = alpha_s * vv - scrh * beta_y;
  if constexpr (D == 3) Rc[Xb][kk] = alpha_s * w - scrh * beta_z;
  Rc[BXt][kk] = dv(-alpha_f * a * beta_y, sqrt_rho);
  if constexpr (D == 3) Rc[BXb][kk] = dv(-alpha_f * a * beta_z, sqrt_rho);
  Rc[ENG][kk] = alpha_s * (Hgas - u * cs) - scrh * beta_v - dv(alpha_f * a * Btmag, sqrt_rho);
  eta[kk] = alpha_s * (X * dV[RHO] + dV[PRS]) - rho * scrh * beta_dv - rho * alpha_s * cs * dV[Xn] -
            sqrt_rho * alpha_f * a * beta_dB;
  eta[kk] *= half_a2;

  kk = KSLOWP;
  lambda[kk] = u + cs;
  Rc[RHO][kk] = alpha_s;
  Rc[Xn][kk] = alpha_s * lambda[kk];
  Rc[Xt][kk] = alpha_s * vv + scrh * beta_y;
  if constexpr (D == 3) Rc[Xb][kk] = alpha_s * w + scrh * beta_z;
  Rc[BXt][kk] = Rc[BXt][KSLOWM];
  if constexpr (D == 3) Rc[BXb][kk] = Rc[BXb][KSLOWM];
  Rc[ENG][kk] = alpha_s * (Hgas + u * cs) + scrh * beta_v - dv(alpha_f * a * Btmag, sqrt_rho);
  eta[kk] = alpha_s * (X * dV[RHO] + dV[PRS]) + rho * scrh * beta_dv + rho * alpha_s * cs * dV[Xn] -
            sqrt_rho * alpha_f * a * beta_dB;
  eta[kk] *= half_a2;

  if constexpr (D == 3) {
    kk = KALFVM;
    lambda[kk] = u - ca;
    Rc[Xt][kk] = -rho * beta_z;
    Rc[Xb][kk] = +rho * beta_y;
    Rc[BXt][kk] = -sBx * sqrt_rho * beta_z;
    Rc[BXb][kk] = sBx * sqrt_rho * beta_y;
    Rc[ENG][kk] = -rho * (vv * beta_z - w * beta_y);
    eta[kk] = +beta_y * dV[Xb] - beta_z * dV[Xt] + dv(sBx, sqrt_rho) * (beta_y * dV[BXb] - beta_z * dV[BXt]);
    eta[kk] *= T(0.5);
    kk = KALFVP;
    lambda[kk] = u + ca;
    Rc[Xt][kk] = -Rc[Xt][KALFVM];
    Rc[Xb][kk] = -Rc[Xb][KALFVM];
    Rc[BXt][kk] = Rc[BXt][KALFVM];
    Rc[BXb][kk] = Rc[BXb][KALFVM];
    Rc[ENG][kk] = -Rc[ENG][KALFVM];
    eta[kk] = -beta_y * dV[Xb] + beta_z * dV[Xt] + dv(sBx, sqrt_rho) * (beta_y * dV[BXb] - beta_z * dV[BXt]);
    eta[kk] *= T(0.5);
  }
  r.cmax = fabs(u) + cf;
  r.sl = lambda[KFASTM];
  r.sr = lambda[KFASTP];
#pragma unroll
  for (int n = 0; n < NV; n++) alambda[n] = fabs(lambda[n]);
  const T hd = T(0.5) * delta, qd = T(0.25) * delta;
  if (alambda[KFASTM] < hd) alambda[KFASTM] = dv(lambda[KFASTM] * lambda[KFASTM], delta) + qd;
  if (alambda[KFASTP] < hd) alambda[KFASTP] = dv(lambda[KFASTP] * lambda[KFASTP], delta) + qd;
  if (alambda[KSLOWM] < hd) alambda[KSLOWM] = dv(lambda[KSLOWM] * lambda[KSLOWM], delta) + qd;
  if (alambda[KSLOWP] < hd) alambda[KSLOWP] = dv(lambda[KSLOWP] * lambda[KSLOWP], delta) + qd;
#pragma unroll
  for (int n1 = 0; n1 < NV; n1++) {
    T s = T(0);
#pragma unroll
    for (int n2 = 0; n2 < NV; n2++) s += alambda[n2] * eta[n2] * Rc[n1][n2];
    r.F[n1] = T(0.5) * (fluxL[n1] + fluxR[n1] - s);
  }
}

template <int D, int DIR, int SOLVER, typename T>
__device__ __forceinline__ void riemann(T gamma, const T* vL, const T* vR, RiemannOut<D, T>& r) {
  if constexpr (SOLVER == kHLLD) riemann_hlld<D, DIR>(gamma, vL, vR, r);
  if constexpr (SOLVER == kHLL) riemann_hll<D, DIR>(gamma, vL, vR, r);
  if constexpr (SOLVER == kROE) riemann_roe<D, DIR>(gamma, vL, vR, r);
  if constexpr (SOLVER == kTVDLF) riemann_tvdlf<D, DIR>(gamma, vL, vR, r);
}

}  // namespace idfx
