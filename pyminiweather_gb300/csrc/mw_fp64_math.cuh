// mw_fp64_math.cuh -- IEEE-FP64 building blocks of the fewest-operation form
// (f64_mode MW_F64_IEEE), shared by its direction-stage kernels
// (mw_fp64_stage.cu) and its adjoint (mw_adjoint.cu).  Every floating-point
// operation on state values is an FP64 add, multiply or FMA; integer
// instructions (bit conversions, table look-ups) are nearly free beside them
// on GB300, whose FP64 pipe retires 2 operations per clock per SM.
#pragma once

#include "mw_common.cuh"

namespace mw {
namespace ieee {

constexpr double binom(double e, int n) {  // C(e, n)
  double c = 1.0;
  for (int k = 0; k < n; ++k) c = c * (e - k) / (k + 1);
  return c;
}
constexpr double cabs(double v) { return v < 0 ? -v : v; }

// The binomial series (1 + d)^e = sum_n C(e, n) d^n: coefficients c[n] and,
// for |d| < 2^-s (s >= 3), the Horner degree deg[s] -- the smallest n with
// |C(e, n+1) / C(e, 1)| 2^(-s n) <= 2^-54, a truncation below half an FP64
// ulp of the first-order term.  |d| >= 1/8 is left to expm1 / log1p.
constexpr int kMaxDeg = 15;
struct Series {
  double c[kMaxDeg + 1];
  unsigned char deg[65];
};
constexpr Series make_series(double e) {
  Series t{};
  for (int n = 0; n <= kMaxDeg; ++n) t.c[n] = binom(e, n);
  for (int s = 0; s <= 64; ++s) {
    int n = kMaxDeg;
    if (s >= 3) {
      for (n = 1; n < kMaxDeg; ++n) {
        double b = cabs(binom(e, n + 1) / binom(e, 1));
        for (int j = 0; j < s * n && b > 0.0; ++j) b *= 0.5;
        if (b <= 5.551115123125783e-17) break;  // 2^-54
      }
    }
    t.deg[s] = (unsigned char)n;
  }
  return t;
}

// An estimate R of 1/y to about 2^-45 without FP64 operations.  With y = m 2^E,
// m in [1, 2), it is formed on the FP32 and integer pipes (which run beside the
// FP64 pipe): the hardware estimate r0 of 1/mh, mh the leading 24 bits of m,
// corrected to first and second order, r1 = r0 (e + e^2), e = 1 - m r0, and
// r0 + r1 put together as a 53-bit integer significand.  far: zero, subnormal,
// Inf, NaN and |y| >= 2^1022, for which R is meaningless.
__device__ __forceinline__ double rcp_estimate(double y, bool& far) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(y);
  const unsigned hi = (unsigned)(b >> 32), lo = (unsigned)b;
  const unsigned ex = (hi >> 20) & 0x7ffu;
  const float mh = __uint_as_float((__funnelshift_l(lo, hi, 3) & 0x007fffffu) | 0x3f800000u);
  const float ml = __uint2float_rn(lo & 0x1fffffffu) * 0x1p-52f;
  float r0;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r0) : "f"(mh));
  const float e0 = fmaf(-ml, r0, fmaf(-mh, r0, 1.0f));
  const int i1 = __float2int_rn(fmaf(e0, e0, e0) * r0 * 0x1p53f);  // |i1| <= 2^31 2^-1
  // R = (M0 2^29 + i1) 2^-53 with r0 = M0 2^-24 in [1/2, 1]: added to the bits of the
  // double r0 2^-E as an integer (a carry or borrow moves the exponent as it should
  // to the accuracy of R)
  const unsigned rb = __float_as_uint(r0);
  const unsigned rhi = (rb >> 3) + ((1919u - ex) << 20);  // 1919 = 1023 + 896: exponent of r0 less that of y
  far = ex - 1u > 2043u;
  return __longlong_as_double((long long)(((unsigned long long)(rhi | (hi & 0x80000000u)) << 32) | (rb << 29)) + i1);
}

// 1/y for the lanes in `mask`, which call it together, in 2 FP64 operations:
// one Newton step from the estimate, r = R + R (1 - y R), squares its error
// (2^-90), so r carries little more than its last rounding.  (A 24-bit
// estimate with a cubic step took 3 operations; the kernels are bound by the
// FP64 pipe, which needs 16 SM clocks per warp operation.)  Where R is
// meaningless the FP64 division is taken, behind a warp-uniform branch so that
// it is never evaluated speculatively on the other lanes.
__device__ __forceinline__ double rcp(double y, unsigned mask) {
  bool far;
  const double R = rcp_estimate(y, far);
  double r = fma(R, fma(-y, R, 1.0), R);
  if (__any_sync(mask, far)) {
    if (far) r = 1.0 / y;
  }
  return r;
}

// N quotients a[k] / y in 3 FP64 operations each, for the lanes in `mask`:
// q = a R, then q + R (a - y q), whose error before the last rounding is 2^-90
// (so it is the correctly rounded quotient but for a few in 2^37).  Quotients
// that leave the normal range, those of -0 (the correction of a zero comes out
// as +0) and divisors with no estimate take the FP64 division.
template <int N>
__device__ __forceinline__ void divide(const double (&a)[N], double y, unsigned mask, double (&q)[N]) {
  bool far;
  const double R = rcp_estimate(y, far);
  const long long y_sign = __double_as_longlong(y) & (long long)0x8000000000000000ull;
#pragma unroll
  for (int k = 0; k < N; ++k) {
    const double q0 = a[k] * R;
    q[k] = fma(R, fma(-y, q0, a[k]), q0);
    // exponents of q and of a within [2^-900, 2^900], or a = 0 and a / y = +0 (integer tests)
    const unsigned eq = (unsigned)(__double_as_longlong(q[k]) >> 52) & 0x7ffu;
    const unsigned ea = (unsigned)(__double_as_longlong(a[k]) >> 52) & 0x7ffu;
    const bool zero = __double_as_longlong(a[k]) == y_sign;
    far = far || (!zero && (eq - 123u > 1800u || ea - 123u > 1800u));
  }
  if (__any_sync(mask, far)) {
    if (far) {
#pragma unroll
      for (int k = 0; k < N; ++k) q[k] = a[k] / y;
    }
  }
}

// The Horner degree of series S that the largest |d| among the lanes in
// `mask` (which call it together) needs; big: this lane's |d| >= 1/8 (or
// Inf / NaN), left out of the degree and to be evaluated otherwise.
__device__ __forceinline__ int series_degree(double d, unsigned mask, const Series& S, bool& big) {
  const unsigned ex = ((unsigned)((unsigned long long)__double_as_longlong(d) >> 52)) & 0x7ffu;
  big = ex >= 1020u;  // |d| >= 2^-3
  const unsigned exm = __reduce_max_sync(mask, big ? 0u : ex);
  const int s = min(1022 - (int)exm, 64);  // |d| < 2^-s for every series lane
  return S.deg[s];
}

// g with (1 + d)^e - 1 = d g: Horner's rule over c[n] .. c[1] (n - 1 FMAs).
__device__ __forceinline__ double series_g(double d, int n, const Series& S) {
  double g = S.c[n];
  for (int k = n - 1; k >= 1; --k) g = fma(g, d, S.c[k]);
  return g;
}

// The stencils of interpolate.py:33-43 and 69-79 by second differences.  With
// t = s(k-1) + s(k+1) every cell gives e = t - 2 s and q = 8 s - t, and the
// interface between cells k - 1 and k has
//   12 x the 4-point interpolation  7 (s(k-1) + s(k)) - (s(k-2) + s(k+1)) = q(k-1) + q(k),
//   the third difference            s(k+1) - s(k-2) + 3 (s(k-1) - s(k))   = e(k) - e(k-1):
// 5 operations per cell and variable where the neighbouring interfaces share
// e and q, against 6 for the two stencils taken one by one.
__device__ __forceinline__ void cell_eq(double sm, double s, double sp, double& e, double& q) {
  const double t = sm + sp;
  e = fma(-2.0, s, t);
  q = fma(8.0, s, -t);
}

// 12 x the 4-point interpolation on its own.
__device__ __forceinline__ double interp12(double s0, double s1, double s2, double s3) {
  return fma(7.0, s1 + s2, -(s0 + s3));
}

}  // namespace ieee
}  // namespace mw
