// mw_f32_flux.cuh -- the FP32 form's arithmetic, shared by the direction kernels
// (mw_f32_dir.cu) and the line kernels (mw_f32_line.cu): the stencils by second
// differences, the variables in packed pairs.  The fluxes are carried as they
// are, not over HV = -2 hv as in the IEEE-FP64 form: HV is no power of two, and
// HV, 1 / HV and the update's factor, each rounded to 24 bits, put the same
// relative error into every flux of a run (rho' after 200 steps at 1024x512:
// 20 % further from FP64), for 2 % of a step (8192x4096: 660 us over HV, 672 as
// they are).
#pragma once

#include "mw_common.cuh"
#include "mw_f32_dir.cuh"
#include "mw_split2.cuh"

namespace mw {
namespace f32 {
namespace {

using split::f2add;
using split::f2fma;
using split::f2mul;
using split::f2splat;
using split::f2sub;

// Constants of one direction of one grid.
struct Consts {
  float HV;              // 2 hv_beta d / (16 dt_full) = -2 hv
  float c[3];            // per stage dt_stage / (2 d)
  float dt[3], gdt[3];   // dt_stage and -dt_stage g
};

// The four variables of a cell (or of a flux).
struct Vars {
  float2 a, b;  // (DENS, UMOM), (WMOM, RHOT)
};
__device__ __forceinline__ float get(const Vars& v, int q) { return q == 0 ? v.a.x : q == 1 ? v.a.y : q == 2 ? v.b.x : v.b.y; }

// Background constants at an interface, times 2 like the interpolated values.
struct Row {
  float R, RT, IRT, P;
};
__device__ __forceinline__ Row row_x(double hyr, double hyrt) {
  const float rt = split::d2f(hyrt);
  return {2.0f * split::d2f(hyr), 2.0f * rt, 0.5f / rt, 2.0f * (float(kC0) * powf(rt, float(kGamma)))};
}
__device__ __forceinline__ Row row_z(double hyr, double hyrt, double hyp) {
  const float rt = split::d2f(hyrt);
  return {2.0f * split::d2f(hyr), 2.0f * rt, 0.5f / rt, 2.0f * split::d2f(hyp)};
}

__device__ __forceinline__ void cell_eq(const Vars& m, const Vars& s, const Vars& p, Vars& e, Vars& q) {
  e.a = f2fma(s.a, f2splat(-2.0f), f2add(m.a, p.a));
  e.b = f2fma(s.b, f2splat(-2.0f), f2add(m.b, p.b));
  q.a = f2fma(e.a, f2splat(-1.0f / 6), s.a);
  q.b = f2fma(e.b, f2splat(-1.0f / 6), s.b);
}

// (1 + d)^gamma - 1: binomial series to degree 6 for |d| <= 1/8 (tail below
// 2^-26 relative); ANY: expm1(gamma log1p(d)) beyond.
template <bool ANY>
__device__ __forceinline__ float pgm1(float d) {
  constexpr double c1 = kGamma, c2 = c1 * (kGamma - 1) / 2, c3 = c2 * (kGamma - 2) / 3, c4 = c3 * (kGamma - 3) / 4,
                   c5 = c4 * (kGamma - 4) / 5, c6 = c5 * (kGamma - 5) / 6;
  float y = fmaf(float(c6), d, float(c5));
  y = fmaf(y, d, float(c4));
  y = fmaf(y, d, float(c3));
  y = fmaf(y, d, float(c2));
  y = fmaf(y, d, float(c1)) * d;
  if (ANY && !(fabsf(d) <= 0.125f)) y = expm1f(float(kGamma) * log1pf(d));
  return y;
}

__device__ __forceinline__ float rcp(float y) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(y));
  return fmaf(r, fmaf(-y, r, 1.0f), r);
}

// Flux times 2 from twice the interpolated values A and the third
// differences D (interpolate.py:82-129, 132-186); w and d3[DENS] vanish at
// walls.  far: set where |d| > 1/8 and ANY is not.
template <int DIR, bool ANY>
__device__ __forceinline__ Vars flux(Vars A, Vars D, const Row& r, const Consts& k, bool wall, bool& far) {
  if (DIR == MW_DIR_Z && wall) {
    A.b.x = 0.0f;
    D.a.x = 0.0f;
  }
  const float m = DIR == MW_DIR_X ? A.a.y : A.b.x;
  const float u = m * rcp(A.a.x + r.R);  // the direction's velocity
  const float d = A.b.y * r.IRT, pp = pgm1<ANY>(d);
  if (!ANY) far = far || !(fabsf(d) <= 0.125f);
  const Vars h = {f2mul(D.a, f2splat(k.HV)), f2mul(D.b, f2splat(k.HV))};  // the hyperviscosity fluxes
  Vars F;
  F.a.x = m + h.a.x;
  if (DIR == MW_DIR_X) {
    F.a.y = fmaf(m, u, fmaf(r.P, pp, h.a.y));
    F.b.x = fmaf(u, A.b.x, h.b.x);
  } else {
    F.a.y = fmaf(u, A.a.y, h.a.y);
    F.b.x = fmaf(m, u, fmaf(r.P, pp, h.b.x));
  }
  F.b.y = fmaf(u, A.b.y + r.RT, h.b.y);
  return F;
}

__device__ __forceinline__ Vars update(const Vars& init, const Vars& Fp, const Vars& F, float c) {
  return {f2fma(f2sub(Fp.a, F.a), f2splat(c), init.a), f2fma(f2sub(Fp.b, F.b), f2splat(c), init.b)};
}

// The same with an increment g of rho w from the source terms: what fluxes and sources add is summed at its
// own scale and the state rounded once (2501x1251: 83.4 -> 85.2 us a step; 8192x4096 the same).
__device__ __forceinline__ Vars update(const Vars& init, const Vars& Fp, const Vars& F, float c, float g) {
  Vars o = update(init, Fp, F, c);
  o.b.x = init.b.x + fmaf(Fp.b.x - F.b.x, c, g);
  return o;
}

// Wall halo of the column value v (ics/bcs.py:92-148): halo row h of -2, -1,
// nz, nz + 1; hr[h] = hyc(halo row) / hyc(wall row).
__device__ __forceinline__ Vars wall_halo(const Vars& v, const double* hr, int h) {
  return {make_float2(v.a.x, (float)((double)v.a.y * hr[h])), make_float2(0.0f, v.b.y)};
}

}  // namespace

// The constants of a direction (d: dx or dz) of a step of size dt.
inline Consts step_consts(double d, double dt_full, double dt) {
  Consts c;
  c.HV = f32_hv(d, dt_full);
  for (int s = 0; s < 3; ++s) {
    c.c[s] = f32_c(d, dt / (3 - s));
    c.dt[s] = (float)(dt / (3 - s));
    c.gdt[s] = c.dt[s] * -float(kGrav);
  }
  return c;
}

}  // namespace f32
}  // namespace mw
