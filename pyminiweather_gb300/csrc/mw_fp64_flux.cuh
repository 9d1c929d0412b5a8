// mw_fp64_flux.cuh -- row constants, pressure and fluxes of the IEEE-FP64 form,
// shared by its direction-stage kernels (mw_fp64_stage.cu) and its line kernels
// (mw_fp64_line.cu).
#pragma once

#include "mw_fp64_math.cuh"

namespace mw {
namespace ieee {

// (1 + d)^gamma: the pressure perturbation.
static __constant__ Series c_pow_g = make_series(kGamma);

// Row constants; the interpolated values are scaled by 12, the fluxes by 12 / HV.
struct RowD {
  double R;      // HV x 12 background rho
  double RT12;   // 12 background rho theta
  double IRT12;  // 1 / (12 background rho theta)
  double P;      // 12 / HV x background pressure C0 (rho theta)^gamma
  double PC1;    // P C(gamma, 1) IRT12: the pressure perturbation per unit of 12 (rho theta)' to first order
};
// HS, IS: HV and 1 / HV times the scale of the interpolated values, 12 (scale, if another).
__device__ __forceinline__ RowD row_consts(double r, double rt, double P, double HS, double IS, double scale = 12.0) {
  const double irt = 1.0 / (scale * rt), p = P * IS;
  return {r * HS, scale * rt, irt, p, p * c_pow_g.c[1] * irt};
}

// P ((1 + d)^gamma - 1) + add, d = AT IRT12, for the lanes in `mask`, which
// call it together: the binomial series to the degree the largest |d| among
// them needs (a warp-uniform loop), or expm1(gamma log1p(d)) for |d| >= 1/8,
// Inf and NaN.  At degree 1 (|d| < 2^-52 on every lane, e.g. a region at
// rest) the series is P C1 d = AT PC1: one FMA in all.
__device__ __forceinline__ double pressure(double AT, const RowD& r, double add, unsigned mask) {
  const double d = AT * r.IRT12;
  bool big;
  const int n = series_degree(d, mask, c_pow_g, big);
  if (n == 1 && !__any_sync(mask, big)) return fma(AT, r.PC1, add);
  double f = d * series_g(d, n, c_pow_g);
  if (__any_sync(mask, big)) {
    if (big) f = expm1(kGamma * log1p(d));
  }
  return fma(r.P, f, add);
}

// Row constants with the pressure series as a polynomial in the interpolated
// 12 (rho theta)' itself: b[n] = P C(gamma, n) IRT12^n, so that
// P ((1 + d)^gamma - 1) = sum_n b[n] AT^n (d = AT IRT12) is Horner's rule in
// AT with no multiplication by IRT12 before it and none by P after it: two
// FP64 operations fewer per interface wherever the degree exceeds one.
struct RowP {
  RowD d;
  double b[kMaxDeg + 1];  // b[0] unused
  int eI;                 // biased exponent of IRT12; 4096 where the b[n] would leave the normal range
  unsigned mI;            // an upper bound of 2^16 x IRT12's significand (in [1, 2)): top 16 fraction bits + 1
};
__device__ __forceinline__ RowP row_consts_p(double r, double rt, double P, double HS, double IS,
                                             double scale = 12.0) {
  RowP o;
  o.d = row_consts(r, rt, P, HS, IS, scale);
  double pw = o.d.IRT12;
  o.b[0] = 0.0;
#pragma unroll
  for (int n = 1; n <= kMaxDeg; ++n) {
    o.b[n] = o.d.P * c_pow_g.c[n] * pw;
    pw *= o.d.IRT12;
  }
  const double lo = fabs(o.b[kMaxDeg]), hi = fabs(o.b[1]);
  const bool normal = fmin(lo, hi) >= 0x1p-1000 && fmax(lo, hi) <= 0x1p1000 && pw >= 0x1p-1000 && pw <= 0x1p1000;
  const unsigned long long bI = (unsigned long long)__double_as_longlong(o.d.IRT12);
  o.eI = normal ? (int)(bI >> 52 & 0x7ffu) : 4096;
  o.mI = (unsigned)(bI >> 36 & 0xffffu) + 0x10001u;
  return o;
}

// The same as pressure(AT, r.d, add, mask), evaluated in AT and to a degree
// chosen per lane, so that a cell's result does not depend on the cells its
// warp happens to hold.  The degree comes from an upper bound on the exponent
// of d = AT IRT12 (the sum of the exponents of AT and IRT12, plus one where the
// product of upper bounds of their leading 17 significand bits reaches 2),
// found by integer operations and never below the degree d itself needs; the
// Horner loop runs from the warp's largest degree, a lane's sum starting (from
// zero) at its own.  Lanes whose bound reaches 1/8 (and Inf, NaN, rows with
// eI = 4096) take the series in d, or expm1 / log1p, at their full degree.
__device__ __forceinline__ double pressure(double AT, const RowP& r, double add, unsigned mask) {
  const unsigned long long bA = (unsigned long long)__double_as_longlong(AT);
  const int exA = (int)(bA >> 52 & 0x7ffu);
  const unsigned mA = (unsigned)(bA >> 36 & 0xffffu) + 0x10001u;
  const int carry = (unsigned long long)mA * r.mI >= (1ull << 33) ? 1 : 0;
  const int eu = exA == 0 ? 0 : exA + r.eI - 1023 + carry;  // biased exponent of d is at most eu
  const bool far = eu >= 1020;
  const int n = far ? 1 : c_pow_g.deg[min(1022 - max(eu, 0), 64)];
  const int nmax = (int)__reduce_max_sync(mask, (unsigned)n);
  double g = n == nmax ? r.b[nmax] : 0.0;
  for (int k = nmax - 1; k >= 1; --k) {
    g = fma(g, AT, r.b[k]);
    if (k > n) g = 0.0;
  }
  double p = fma(g, AT, add);
  if (__any_sync(mask, far)) {
    if (far) {
      const double d = AT * r.d.IRT12;
      const bool big = !(fabs(d) < 0.125);
      double f = d * series_g(d, kMaxDeg, c_pow_g);
      if (big) f = expm1(kGamma * log1p(d));
      p = fma(r.d.P, f, add);
    }
  }
  return p;
}

__device__ __forceinline__ const RowD& rowd(const RowD& r) { return r; }
__device__ __forceinline__ const RowD& rowd(const RowP& r) { return r.d; }

// x flux times 12 / HV (interpolate.py:82-129) from 12 x the interpolated
// values A and the third differences D: with u = (rho u)' / rho,
// F = ((rho u)', u (rho u)' + p', u (rho w)', u (rho theta)) - hv d3, HV = -12 hv.
template <typename Row>
__device__ __forceinline__ void flux_x(const double A[4], const double D[4], const Row& r, double HV, double IHV,
                                       unsigned mask, double F[4]) {
  const double u = A[UMOM] * rcp(fma(HV, A[DENS], rowd(r).R), mask);  // u / HV
  F[0] = fma(IHV, A[UMOM], D[DENS]);
  F[1] = fma(A[UMOM], u, pressure(A[RHOT], r, D[UMOM], mask));
  F[2] = fma(u, A[WMOM], D[WMOM]);
  F[3] = fma(u, A[RHOT] + rowd(r).RT12, D[RHOT]);
}

// z flux times 12 / HV (interpolate.py:132-186); w and d3[DENS] vanish at the walls.
template <typename Row>
__device__ __forceinline__ void flux_z(const double A[4], const double D[4], const Row& r, double HV, double IHV,
                                       bool wall, unsigned mask, double F[4]) {
  const double AW = wall ? 0.0 : A[WMOM];
  const double w = AW * rcp(fma(HV, A[DENS], rowd(r).R), mask);  // w / HV
  F[0] = fma(IHV, AW, wall ? 0.0 : D[DENS]);
  F[1] = fma(w, A[UMOM], D[UMOM]);
  F[2] = fma(AW, w, pressure(A[RHOT], r, D[WMOM], mask));
  F[3] = fma(w, A[RHOT] + rowd(r).RT12, D[RHOT]);
}

}  // namespace ieee
}  // namespace mw
