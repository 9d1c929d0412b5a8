// mw_adjoint.cu -- adjoint (vector-Jacobian product) of one direction-stage.
//
// Forward (pyminiweather/solve/step.py:21-82, interpolate.py:82-250):
//   out = init + dt * L(forcing),  L = -(F(i+1) - F(i)) / d  [- rho' g on w in z],
//   F(i) = f(A(i), D(i)),  A = sum_j c_j s(i-2+j),  D = sum_j e_j s(i-2+j),
//   c = (-1, 7, 7, -1)/12, e = (-1, 3, -3, 1), s read through the halo rules
//   (periodic in x, ics/bcs.py:35-39; wall in z, bcs.py:92-148).
// Adjoint, given g = dJ/d(out) on the interior cells:
//   dJ/d(init)    += g
//   dJ/d(forcing) += dt * (dL/d forcing)^T g:
//     Fbar(i) = (dt/d) (g(i) - g(i-1))      (g = 0 outside the interior)
//     (Abar, Dbar)(i) = (df/dA, df/dD)^T Fbar(i)
//     sbar(t) += c_j Abar(i) + e_j Dbar(i)  for the taps t = i-2+j, mapped
//     back through the halo rules (a halo value's adjoint goes to the cell it
//     was copied or scaled from), and sbar_rho(k) -= dt g_w(k) grav in z.
// The flux Jacobian uses rho theta = A3 + (rho theta)_bg and p = C0 (rho theta)^gamma,
// so dp/dA3 = gamma p / (rho theta); at the z walls w and d3[DENS] are held at
// zero (interpolate.py:167-173), so those paths carry no adjoint.
//
// f64_mode MW_F64_NATIVE (the reference's formulas: a pow and three divides
// per interface) runs two kernels per call: one thread per interface writes
// (Abar, Dbar) to a caller-provided workspace; one thread per cell gathers its
// taps.  MW_F64_IEEE (the fewest FP64 operations: values scaled by 12, 1/rho
// by a Newton step, dp/d(rho theta) = gamma P_row (1 + delta)^(gamma-1) /
// (rho theta)_bg by its binomial series, per-row constants from a table in the
// workspace) runs one kernel in either direction, which computes the interface
// adjoints of a warp's segment (x) or a CTA's tile (z) into shared memory and
// gathers them there.
#include <algorithm>

#include "mw_common.cuh"
#include "mw_fp64_math.cuh"
#include "mw_pow.cuh"

namespace mw {
namespace {

struct VjpArgs {
  int nx, nz, pitch;
  long long plane;
  double d;         // dx or dz
  double hv;        // -hv_beta d / (16 dt_full)
  double dt_stage;
  const double *hyc, *hytc, *hyi, *hyti, *hypi;
  const double* forcing;
  const double* gout;
  const double* base_a;
  const double* base_b;
  int add_gout;
  double* gdst;
  double* ws;       // 8 x n_interfaces: Abar[4], Dbar[4]
  long long nif;    // interfaces per variable plane of ws
  double kc, ke;    // IEEE form: the gather's factors of the transposed interpolation (of 12 x it, over 12) and third
                    // difference, which its interface adjoints do not carry
};

__device__ __forceinline__ int wrap_x(int j, int nx) { return j < 0 ? j + nx : (j >= nx ? j - nx : j); }

// Bounds-checked element access (MW_AT) to the arrays of one stage adjoint.
#define MW_VF(a, off) MW_AT((a).forcing, (off), 4 * (a).plane)
#define MW_VC(a, p, k) MW_AT((a).p, (k), (a).nz + 2 * kHs)  // cell-centre background
#define MW_VI(a, p, k) MW_AT((a).p, (k), (a).nz + 1)        // interface background
#define MW_WS(a, off) MW_AT((a).ws, (off), 8 * (a).nif)

__device__ __forceinline__ double zval(const VjpArgs& a, int q, int k, int col) {
  if (k >= 0 && k < a.nz) return MW_VF(a, q * a.plane + (long long)(k + kHs) * a.pitch + col);
  if (q == WMOM) return 0.0;
  const int src = k < 0 ? kHs : a.nz + kHs - 1;
  const double s = MW_VF(a, q * a.plane + (long long)src * a.pitch + col);
  if (q == UMOM) return s / MW_VC(a, hyc, src) * MW_VC(a, hyc, k + kHs);
  return s;
}

__device__ __forceinline__ double gval(const VjpArgs& a, int q, int k, int i) {
  return MW_AT(a.gout, q * a.plane + (long long)(k + kHs) * a.pitch + i + kHs, 4 * a.plane);
}

// tap weights of the interpolation (data/fields.py:94-97, convolution order
// reversed) and of the third difference
__constant__ double kC[4] = {-1.0 / 12, 7.0 / 12, 7.0 / 12, -1.0 / 12};
__constant__ double kE[4] = {-1.0, 3.0, -3.0, 1.0};

// Interface adjoints.  x: interface (k, i), i in [0, nx]; z: (k, c), k in [0, nz].
template <int DIR>
__global__ void k_vjp_iface(VjpArgs a) {
  overlap_wait();
  const long long n = a.nif;
  for (long long idx = blockIdx.x * (long long)blockDim.x + threadIdx.x; idx < n;
       idx += (long long)gridDim.x * blockDim.x) {
    double s[4][4];
    double Fb[4];
    bool wall = false;
    double hy_r, hy_rt;
    if (DIR == MW_DIR_X) {
      const int k = (int)(idx / (a.nx + 1)), i = (int)(idx % (a.nx + 1));
      const long long row = (long long)(k + kHs) * a.pitch;
      for (int j = 0; j < 4; ++j) {
        const long long col = wrap_x(i - 2 + j, a.nx) + kHs;
        for (int q = 0; q < 4; ++q) s[q][j] = MW_VF(a, q * a.plane + row + col);
      }
      for (int q = 0; q < 4; ++q) {
        const double gr = i < a.nx ? gval(a, q, k, i) : 0.0;
        const double gl = i > 0 ? gval(a, q, k, i - 1) : 0.0;
        Fb[q] = a.dt_stage / a.d * (gr - gl);
      }
      hy_r = MW_VC(a, hyc, k + kHs);
      hy_rt = MW_VC(a, hytc, k + kHs);
    } else {
      const int k = (int)(idx / a.nx), c = (int)(idx % a.nx);
      for (int j = 0; j < 4; ++j)
        for (int q = 0; q < 4; ++q) s[q][j] = zval(a, q, k - 2 + j, c + kHs);
      for (int q = 0; q < 4; ++q) {
        const double gr = k < a.nz ? gval(a, q, k, c) : 0.0;
        const double gl = k > 0 ? gval(a, q, k - 1, c) : 0.0;
        Fb[q] = a.dt_stage / a.d * (gr - gl);
      }
      hy_r = MW_VI(a, hyi, k);
      hy_rt = MW_VI(a, hyti, k);
      wall = (k == 0) || (k == a.nz);
    }
    double A[4];
    for (int q = 0; q < 4; ++q) A[q] = ((s[q][0] * kC[0] + s[q][1] * kC[1]) + s[q][2] * kC[2]) + s[q][3] * kC[3];
    const double rho = A[DENS] + hy_r;
    const double rt = A[RHOT] + hy_rt;
    const double u = A[UMOM] / rho, w = A[WMOM] / rho, th = rt / rho;
    const double dpdA3 = kGamma * kC0 * pow(rt, kGamma) / rt;
    double Ab[4], Db[4];
    for (int q = 0; q < 4; ++q) Db[q] = -a.hv * Fb[q];
    if (DIR == MW_DIR_X) {
      Ab[DENS] = -(Fb[1] * u * u + Fb[2] * u * w + Fb[3] * u * th);
      Ab[UMOM] = Fb[0] + 2.0 * Fb[1] * u + Fb[2] * w + Fb[3] * th;
      Ab[WMOM] = Fb[2] * u;
      Ab[RHOT] = Fb[1] * dpdA3 + Fb[3] * u;
    } else if (!wall) {
      Ab[DENS] = -(Fb[1] * w * u + Fb[2] * w * w + Fb[3] * w * th);
      Ab[UMOM] = Fb[1] * w;
      Ab[WMOM] = Fb[0] + Fb[1] * u + 2.0 * Fb[2] * w + Fb[3] * th;
      Ab[RHOT] = Fb[2] * dpdA3 + Fb[3] * w;
    } else {
      Ab[DENS] = 0.0;
      Ab[UMOM] = 0.0;
      Ab[WMOM] = 0.0;
      Ab[RHOT] = Fb[2] * dpdA3;
      Db[DENS] = 0.0;
    }
    for (int q = 0; q < 4; ++q) {
      MW_WS(a, q * n + idx) = Ab[q];
      MW_WS(a, (4 + q) * n + idx) = Db[q];
    }
  }
}

// g_dst of one value from its gathered adjoint: + g_out (add_gout), + the bases, which may be far larger, last.
__device__ __forceinline__ void store_value(const VjpArgs& a, long long oq, double v) {
  if (a.add_gout) v += MW_AT(a.gout, oq, 4 * a.plane);
  if (a.base_a) v += MW_AT(a.base_a, oq, 4 * a.plane);
  if (a.base_b) v += MW_AT(a.base_b, oq, 4 * a.plane);
  MW_AT(a.gdst, oq, 4 * a.plane) = v;
}

// Cell gather: gdst = base_a + base_b + add_gout * gout + sbar (interior); halo cells of gdst = 0.
// The adjoint of interior cell (k, i) gathered from the interface adjoints
// of its taps by the general rule: periodic wrap in x, the wall rule's halo
// taps in z (any cell).
template <int DIR>
__device__ __forceinline__ void gather_general(const VjpArgs& a, int k, int i, double acc[4]) {
  const long long n = a.nif;
  auto tap = [&](int q, int j, long long o) {
    return kC[j] * MW_WS(a, q * n + o) + kE[j] * MW_WS(a, (4 + q) * n + o);
  };
  if (DIR == MW_DIR_X) {
    for (int j = 0; j < 4; ++j)
      for (int m = -1; m <= 1; ++m) {
        const int f = i + 2 - j + m * a.nx;  // interface whose tap j is cell i
        if (f < 0 || f > a.nx) continue;
        const long long o = (long long)k * (a.nx + 1) + f;
        for (int q = 0; q < 4; ++q) acc[q] += tap(q, j, o);
      }
  } else {
    // taps t = f - 2 + j of interface f in [0, nz]; t maps to row k directly,
    // or through the wall rule from halo rows -2,-1 (-> 0) and nz, nz+1 (-> nz-1)
    for (int f = k - 1; f <= k + 2; ++f) {  // interfaces with an interior tap at row k
      if (f < 0 || f > a.nz) continue;
      const int j = k - f + 2;
      const long long o = (long long)f * a.nx + i;
      for (int q = 0; q < 4; ++q) acc[q] += tap(q, j, o);
    }
    auto halo_taps = [&](int t, double wq[4]) {  // weight of halo row t on row k
      const int src = t < 0 ? 0 : a.nz - 1;
      wq[DENS] = wq[RHOT] = (k == src) ? 1.0 : 0.0;
      wq[WMOM] = 0.0;
      wq[UMOM] = (k == src) ? MW_VC(a, hyc, t + kHs) / MW_VC(a, hyc, src + kHs) : 0.0;
    };
    const int halo_rows[4] = {-2, -1, a.nz, a.nz + 1};
    for (int h = 0; h < 4; ++h) {
      const int t = halo_rows[h];
      double wq[4];
      halo_taps(t, wq);
      if (wq[DENS] == 0.0 && wq[UMOM] == 0.0) continue;
      for (int j = 0; j < 4; ++j) {
        const int f = t + 2 - j;
        if (f < 0 || f > a.nz) continue;
        const long long o = (long long)f * a.nx + i;
        for (int q = 0; q < 4; ++q)
          acc[q] += wq[q] * tap(q, j, o);
      }
    }
  }
}

// One thread per cell of a row (grid.y strides over the rows): halo cells get
// zero; an interior cell whose four interfaces are all interior and none of
// whose taps wrap or come through the wall rule (x: 2 <= i <= nx - 3, z:
// 1 <= k <= nz - 2) reads them as a row (x) or column (z) of four, A0 .. A3
// and D0 .. D3 at interfaces i - 1 .. i + 2, and sums the transposed taps in
// the symmetric forms (7 (A1 + A2) - (A0 + A3)) / 12 and (D0 - D3) + 3 (D2 - D1);
// the others take the general rule.  In z the gravity term follows.
template <int DIR>
__global__ void __launch_bounds__(128) k_vjp_gather(VjpArgs a) {
  overlap_wait();
  const long long n = a.nif;
  const int ii = blockIdx.x * blockDim.x + threadIdx.x;
  if (ii >= a.pitch) return;
  const int i = ii - kHs;
  for (int kk = blockIdx.y; kk < a.nz + 2 * kHs; kk += gridDim.y) {
    const long long idx = (long long)kk * a.pitch + ii;
    const int k = kk - kHs;
    if (k < 0 || k >= a.nz || i < 0 || i >= a.nx) {
      for (int q = 0; q < 4; ++q) MW_AT(a.gdst, q * a.plane + idx, 4 * a.plane) = 0.0;
      continue;
    }
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    const bool fast = DIR == MW_DIR_X ? (i >= 2 && i + 3 <= a.nx) : (k >= 1 && k + 2 <= a.nz);
    if (fast) {
      // interfaces i - 1 .. i + 2 (x: row k of nx + 1; z: rows k - 1 .. k + 2 of column i)
      const long long o0 = DIR == MW_DIR_X ? (long long)k * (a.nx + 1) + (i - 1) : (long long)(k - 1) * a.nx + i;
      const long long st = DIR == MW_DIR_X ? 1 : a.nx;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double A0 = MW_WS(a, q * n + o0), A1 = MW_WS(a, q * n + o0 + st);
        const double A2 = MW_WS(a, q * n + o0 + 2 * st), A3 = MW_WS(a, q * n + o0 + 3 * st);
        const double D0 = MW_WS(a, (4 + q) * n + o0), D1 = MW_WS(a, (4 + q) * n + o0 + st);
        const double D2 = MW_WS(a, (4 + q) * n + o0 + 2 * st), D3 = MW_WS(a, (4 + q) * n + o0 + 3 * st);
        // cell i is tap j of interface f = i + 2 - j, so kC = (-1, 7, 7, -1) / 12 and
        // kE = (-1, 3, -3, 1) act on the interfaces i + 2, i + 1, i, i - 1 = (A3, A2, A1, A0)
        const double ca = fma(7.0, A1 + A2, -(A0 + A3)) * (1.0 / 12.0);
        const double ce = fma(3.0, D2 - D1, D0 - D3);
        acc[q] = ca + ce;
      }
    } else {
      gather_general<DIR>(a, k, i, acc);
    }
    if (DIR == MW_DIR_Z) acc[DENS] -= a.dt_stage * kGrav * gval(a, WMOM, k, i);
    for (int q = 0; q < 4; ++q) store_value(a, q * a.plane + idx, acc[q]);
  }
}

// ---- IEEE-FP64 interface adjoint (f64_mode MW_F64_IEEE) --------------------
__constant__ ieee::Series c_pow_gm1 = ieee::make_series(kGamma - 1.0);  // (1 + d)^(gamma - 1)

// Row constants of the IEEE interface adjoint, scaled by 12 like the
// interpolated values: the x rows (cell centres, nz + 4 entries), then the z
// interface rows (nz + 1), in the workspace after the interface adjoints.
struct RowV {
  double R12;    // 12 background rho
  double RT12;   // 12 background rho theta
  double IRT12;  // 1 / (12 background rho theta)
  double Q;      // dp/d(rho theta) at the background, gamma C0 (rho theta)^(gamma - 1)
  double QC1;    // Q C(gamma - 1, 1) IRT12: its change per unit of 12 (rho theta)' to first order
};

__global__ void k_vjp_rows_ieee(int nz, const double* hyc, const double* hytc, const double* hyi, const double* hyti,
                                const double* hypi, RowV* t) {
  __shared__ PowTables pow_tables;
  load_pow_tables(pow_tables);
  __syncthreads();
  const int n = 2 * nz + 5;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
    double r, rt, Q;
    if (j < nz + 2 * kHs) {
      r = MW_AT(hyc, j, nz + 2 * kHs);
      rt = MW_AT(hytc, j, nz + 2 * kHs);
      Q = kGamma * (kC0 * pow_gamma(rt, pow_tables)) / rt;  // gamma C0 (rho theta)^(gamma - 1)
    } else {  // hy_pressure_int = C0 hy_dens_theta_int^gamma (ics/initial.py:105)
      const int k = j - (nz + 2 * kHs);
      r = MW_AT(hyi, k, nz + 1);
      rt = MW_AT(hyti, k, nz + 1);
      Q = kGamma * MW_AT(hypi, k, nz + 1) / rt;
    }
    const double irt = 1.0 / (12.0 * rt);
    MW_AT(t, j, n) = {12.0 * r, 12.0 * rt, irt, Q, Q * c_pow_gm1.c[1] * irt};
  }
}

// J(f)^T of one interface in the fewest FP64 operations (~35 against ~300
// for k_vjp_iface, the same Jacobian): taps s, G = g(f) - g(f-1), the row
// constants rv; Ab = J^T G and Db = G (the gather applies their factors cd and
// hvcd), with (rho w)' and d3[DENS] held at zero at the z walls.  The lanes in
// `mask` call it together.
template <int DIR>
__device__ __forceinline__ void jt_ieee(const double s[4][4], const double Fb[4], const RowV& rv, bool wall,
                                        unsigned mask, double Ab[4], double Db[4]) {
  double A[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) A[q] = ieee::interp12(s[q][0], s[q][1], s[q][2], s[q][3]);
  const double ri = ieee::rcp(A[DENS] + rv.R12, mask);
  const double u = A[UMOM] * ri, w = A[WMOM] * ri, th = (A[RHOT] + rv.RT12) * ri;
  // dp/dA3 = Q (1 + d)^(gamma - 1), d = (rho theta)' / (rho theta)_bg
  const double d = A[RHOT] * rv.IRT12;
  bool big;
  const int deg = ieee::series_degree(d, mask, c_pow_gm1, big);
  double dp;
  if (deg == 1 && !__any_sync(mask, big)) {
    dp = fma(A[RHOT], rv.QC1, rv.Q);
  } else {
    dp = fma(rv.Q * d, ieee::series_g(d, deg, c_pow_gm1), rv.Q);
    if (__any_sync(mask, big)) {
      if (big) dp = rv.Q * exp((kGamma - 1.0) * log1p(d));
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) Db[q] = Fb[q];
  if (DIR == MW_DIR_X) {
    const double y = fma(Fb[1], u, fma(Fb[2], w, Fb[3] * th));  // Fb1 u + Fb2 w + Fb3 th
    Ab[DENS] = -(u * y);
    Ab[UMOM] = fma(Fb[1], u, Fb[0]) + y;
    Ab[WMOM] = Fb[2] * u;
    Ab[RHOT] = fma(Fb[1], dp, Fb[3] * u);
  } else if (!wall) {
    const double y = fma(Fb[1], u, fma(Fb[2], w, Fb[3] * th));
    Ab[DENS] = -(w * y);
    Ab[UMOM] = Fb[1] * w;
    Ab[WMOM] = fma(Fb[2], w, Fb[0]) + y;
    Ab[RHOT] = fma(Fb[2], dp, Fb[3] * w);
  } else {
    Ab[DENS] = 0.0;
    Ab[UMOM] = 0.0;
    Ab[WMOM] = 0.0;
    Ab[RHOT] = Fb[2] * dp;
    Db[DENS] = 0.0;
  }
}

// ---- IEEE-FP64 stage adjoint, x: one kernel ---------------------------------
// The interface adjoints (jt_ieee) and the gather of their transposed taps in
// one pass, with no round trip through the workspace: a warp walks 29-cell
// segments of a row; lane l computes interface f = p0-1+l into shared memory
// and, for l < 29, gathers cell p0+l from interfaces p0-1+l .. p0+2+l in the
// symmetric forms of k_vjp_gather.  The row is periodic: interface f takes its
// taps and G = g(f) - g(f-1) with the periodic rule, so the reference's
// interfaces 0 and nx, which share their taps, enter as one.
constexpr int kFVCells = 29;
constexpr int kFVPos = kFVCells + 6;  // forcing positions p0-3 .. p0+31
constexpr int kFXThreads = 256;
constexpr int kFXWarps = kFXThreads / 32;

struct SmemFX {
  double s[kFXWarps][4][kFVPos];  // forcing at positions p0-3 .. p0+31
  double g[kFXWarps][4][33];      // g at positions p0-2 .. p0+30
  double ab[kFXWarps][4][32];     // Ab at interfaces p0-1 .. p0+30
  double db[kFXWarps][4][32];     // Db
};

// The transposed taps of interface adjoints A0 .. A3, D0 .. D3 (interfaces i - 1 .. i + 2) on cell i.
__device__ __forceinline__ double gather4(const VjpArgs& a, double A0, double A1, double A2, double A3, double D0,
                                          double D1, double D2, double D3) {
  const double ca = fma(7.0, A1 + A2, -(A0 + A3));
  const double ce = fma(3.0, D2 - D1, D0 - D3);
  return fma(a.kc * (1.0 / 12.0), ca, a.ke * ce);
}

__global__ void __launch_bounds__(kFXThreads) k_vjp_ieee_x(VjpArgs a, const RowV* rows, int nseg, long long total) {
  __shared__ SmemFX sm;
  overlap_wait();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long b0 = total * blockIdx.x / gridDim.x, b1 = total * (blockIdx.x + 1) / gridDim.x;
  const long long g0 = b0 + (b1 - b0) * w / kFXWarps, g1 = b0 + (b1 - b0) * (w + 1) / kFXWarps;
  auto col = [&](int p) { return ((p % a.nx) + a.nx) % a.nx + kHs; };  // periodic
  for (long long g = g0; g < g1; ++g) {
    const int k = (int)(g / nseg), p0 = (int)(g - (long long)k * nseg) * kFVCells;
    const long long row = (long long)(k + kHs) * a.pitch;
    {
      const int cA = col(p0 - 3 + lane), cB = col(p0 + 29 + lane), cG = col(p0 - 1 + lane), cH = col(p0 - 2);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        sm.s[w][q][lane] = MW_VF(a, q * a.plane + row + cA);
        if (lane < 3) sm.s[w][q][32 + lane] = MW_VF(a, q * a.plane + row + cB);
        sm.g[w][q][lane + 1] = MW_AT(a.gout, q * a.plane + row + cG, 4 * a.plane);
        if (lane == 0) sm.g[w][q][0] = MW_AT(a.gout, q * a.plane + row + cH, 4 * a.plane);
      }
    }
    __syncwarp();
    {  // interface f = p0 - 1 + lane
      double s[4][4], dg[4], Ab[4], Db[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int j = 0; j < 4; ++j) s[q][j] = sm.s[w][q][lane + j];
        dg[q] = sm.g[w][q][lane + 1] - sm.g[w][q][lane];
      }
      const RowV rv = MW_AT(rows, k + kHs, 2 * a.nz + 5);
      jt_ieee<MW_DIR_X>(s, dg, rv, false, 0xffffffffu, Ab, Db);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        sm.ab[w][q][lane] = Ab[q];
        sm.db[w][q][lane] = Db[q];
      }
    }
    __syncwarp();
    const int t = p0 + lane;  // cell
    if (lane < kFVCells && t < a.nx) {
      double acc[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double* ab = sm.ab[w][q] + lane;
        const double* db = sm.db[w][q] + lane;
        acc[q] = gather4(a, ab[0], ab[1], ab[2], ab[3], db[0], db[1], db[2], db[3]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) store_value(a, q * a.plane + row + t + kHs, acc[q]);
    }
    __syncwarp();
  }
  zero_frame(a.gdst, a.nx, a.nz, a.plane);
}

// ---- IEEE-FP64 stage adjoint, z: one kernel ---------------------------------
// A CTA takes 2^LC columns (32; fewer on narrow grids, more on flat ones) of up
// to fz_max_rows(LC) rows.  Its threads, 2^LC to a stretch, first compute the
// tile's rows + 3 interface adjoints, each a stretch of consecutive interfaces
// down its column (the four taps and g move along in registers, one new row of
// each per interface), into shared memory; then, after the one barrier, each
// gathers a stretch of rows the same way (one new interface per row).
//
// Bound: FP64 (512 x 256, a stage without bases: 2375 instructions on the
// fullest SM at 16 cycles each, 38000 of its 53500 active cycles; the rest is
// the first and last loads and stores, which all warps meet together).  29.7 us
// a stage at 512 x 256, with the bases counted in, against 14.8 + 21 us for
// the interface adjoints and the gather as two kernels with the 8 values per
// interface in memory between them.  Sixteen warps a CTA: 33 us.  Rows read
// one interface ahead: no gain.
constexpr int kFZThreads = 256;
constexpr int kFZWarps = kFZThreads / 32;

// 64 KB of shared memory: 32 interfaces of 32 columns
__host__ __device__ constexpr int fz_max_rows(int lc) { return (1024 >> lc) - 3; }
static_assert(fz_max_rows(7) >= 5, "the widest tile");
inline int fz_smem(int rows, int lc) { return ((int)sizeof(double) * 8 * (rows + 3)) << lc; }

// The wall rule's halo taps on row k (0 or nz - 1, or both): halo row t passes weight wq of its adjoint to row `src`.
template <int C>
__device__ __forceinline__ void gather_wall(const VjpArgs& a, const double* ws, int f0, int k, double acc[4]) {
  for (int t = -2; t <= a.nz + 1; t = t == -1 ? a.nz : t + 1) {
    const int src = t < 0 ? 0 : a.nz - 1;
    if (src != k) continue;
    const double wu = MW_VC(a, hyc, t + kHs) / MW_VC(a, hyc, src + kHs);
    for (int j = 0; j < 4; ++j) {
      const int f = t + 2 - j;
      if (f < 0 || f > a.nz) continue;
      const double* c = ws + (f - f0) * 8 * C;
      for (int q = 0; q < 4; ++q) {
        if (q == WMOM) continue;
        acc[q] += (q == UMOM ? wu : 1.0) * (a.kc * (kC[j] * c[q * C]) + a.ke * (kE[j] * c[(4 + q) * C]));
      }
    }
  }
}

// g_dst of a cell (offset o in a plane).  With g_out and both bases, as in the last stage of a direction, the twelve
// loads are in flight together: one by one behind the stores the few warps of a tile waited for each (31.1 us a stage
// on average, 29.7 so; the x kernel, with twice the warps, is slower so: 27.3 against 29.1).
__device__ __forceinline__ void store_cell(const VjpArgs& a, long long o, const double acc[4]) {
  if (a.add_gout && a.base_a && a.base_b) {
    double g[4], p[4], r[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      g[q] = MW_AT(a.gout, q * a.plane + o, 4 * a.plane);
      p[q] = MW_AT(a.base_a, q * a.plane + o, 4 * a.plane);
      r[q] = MW_AT(a.base_b, q * a.plane + o, 4 * a.plane);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) MW_AT(a.gdst, q * a.plane + o, 4 * a.plane) = acc[q] + g[q] + p[q] + r[q];
    return;
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) store_value(a, q * a.plane + o, acc[q]);
}

template <int LC>
__global__ void __launch_bounds__(kFZThreads) k_vjp_ieee_z(VjpArgs a, const RowV* rows, int tile_rows) {
  extern __shared__ double fz_ws[];  // [interface][Ab 0..3, Db 0..3][column]
  constexpr int C = 1 << LC, S = kFZWarps * 32 / C;  // columns and stretches of a tile
  overlap_wait();
  const int lane = threadIdx.x & (C - 1), w = threadIdx.x >> LC;  // column and stretch of the thread
  const int nxt = (a.nx + C - 1) / C, nzt = (a.nz + tile_rows - 1) / tile_rows;
  for (long long tile = blockIdx.x; tile < (long long)nxt * nzt; tile += gridDim.x) {
    const int k0 = (int)(tile / nxt) * tile_rows, k1 = min(a.nz, k0 + tile_rows);
    const int c = (int)(tile % nxt) * C + lane;
    const bool in = c < a.nx;
    const int col = min(c, a.nx - 1) + kHs;  // columns past the grid repeat the last one and are not stored
    const int fa = max(0, k0 - 1), fb = min(a.nz, k1 + 1);  // interfaces fa .. fb
    double* ws = fz_ws + lane;
    {
      const int n = fb - fa + 1, f0 = fa + n * w / S, f1 = fa + n * (w + 1) / S;
      // the lanes of a warp go together: a stretch that is one interface shorter, or empty, ends on one that is not its
      // own (and not stored)
      const int end = LC >= 5 ? f1 : f0 + (n + S - 1) / S;
      double s[4][4], gl[4];
      if (f0 < end) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
          for (int j = 1; j < 4; ++j) s[q][j] = zval(a, q, f0 - 3 + j, col);
          gl[q] = f0 > 0 ? gval(a, q, f0 - 1, col - kHs) : 0.0;
        }
      }
      for (int i = f0; i < end; ++i) {
        const int f = LC >= 5 ? i : min(i, fb);
        double dg[4], Ab[4], Db[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          s[q][0] = s[q][1];
          s[q][1] = s[q][2];
          s[q][2] = s[q][3];
          s[q][3] = zval(a, q, f + 1, col);
          const double gr = f < a.nz ? gval(a, q, f, col - kHs) : 0.0;
          dg[q] = gr - gl[q];
          gl[q] = gr;
        }
        const RowV rv = MW_AT(rows, a.nz + 2 * kHs + f, 2 * a.nz + 5);
        jt_ieee<MW_DIR_Z>(s, dg, rv, f == 0 || f == a.nz, 0xffffffffu, Ab, Db);
        if (LC >= 5 || i < f1) {
          double* o = ws + (f - fa) * 8 * C;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            o[q * C] = Ab[q];
            o[(4 + q) * C] = Db[q];
          }
        }
      }
    }
    __syncthreads();
    {
      const int n = k1 - k0, r0 = k0 + n * w / S, r1 = k0 + n * (w + 1) / S;
      double A[4][4], D[4][4];
      // interface f of the tile; one outside [0, nz] has no adjoint
      auto load = [&](int f, int j) {
        const bool has = f >= 0 && f <= a.nz;
        const double* p = ws + (f - fa) * 8 * C;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          A[q][j] = has ? p[q * C] : 0.0;
          D[q][j] = has ? p[(4 + q) * C] : 0.0;
        }
      };
      if (r0 < r1) {
        load(r0 - 1, 1);
        load(r0, 2);
        load(r0 + 1, 3);
      }
      for (int k = r0; k < r1; ++k) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            A[q][j] = A[q][j + 1];
            D[q][j] = D[q][j + 1];
          }
        load(k + 2, 3);
        double acc[4];
        const long long o = (long long)(k + kHs) * a.pitch + col;
#pragma unroll
        for (int q = 0; q < 4; ++q)
          acc[q] = gather4(a, A[q][0], A[q][1], A[q][2], A[q][3], D[q][0], D[q][1], D[q][2], D[q][3]);
        if (k == 0 || k == a.nz - 1) gather_wall<C>(a, ws, fa, k, acc);
        acc[DENS] = fma(-a.dt_stage * kGrav, gval(a, WMOM, k, col - kHs), acc[DENS]);
        if (in) store_cell(a, o, acc);
      }
    }
    __syncthreads();
  }
  zero_frame(a.gdst, a.nx, a.nz, a.plane);
}

// Columns (log2) and rows of a tile of k_vjp_ieee_z: those with the fewest rounds
// of a warp's work, interfaces and rows counted alike (about 40 FP64 operations
// each) and one more per tile for its loads, on the SM with the most tiles; of
// equals the tallest, which recompute the fewest interfaces.  512 x 256: 29 rows,
// 144 tiles, 29.7 us.  From a third to twice the charge per tile: the same times
// within 1 % from 100 x 50 to 640 x 448.  Grids of fewer than 256 columns, where
// tiles of 32 may leave a good part of the lanes idle, may take narrower tiles
// (a stage, us in tiles of 32 and as chosen: 8x20000 145, 64; 2x100000 594, 78;
// 66x9000 189, 153), grids of fewer rows than warps wider ones (3000000x2 2950, 2170).
struct FzTile {
  int lc, rows;
};
inline FzTile fz_tile(int nx, int nz, int sms) {
  FzTile best = {5, std::min(nz, fz_max_rows(5))};
  double cost = 0;
  const int widths[] = {5, 4, 3, 2, 1, 6, 7};
  for (const int lc : widths) {
    if (lc < 5 ? nx >= 256 : lc > 5 && nz >= kFZWarps) continue;
    const long long nxt = (nx + (1 << lc) - 1) >> lc;
    const int S = kFZWarps * 32 >> lc, step = lc >= 5 ? 1 : S, most = std::min(nz, fz_max_rows(lc));
    // rows such that rows + 3 interfaces are whole rounds of the stretches
    for (int r = lc >= 5 ? 1 : std::min(S - 3, most); r <= most; r += step) {
      const long long nzt = (nz + r - 1) / r, per_sm = (nxt * nzt + sms - 1) / sms;
      const double c = per_sm * ((std::min(r + 3, nz + 1) + S - 1) / S + (r + S - 1) / S + 1.0);
      // the tallest of a width; another width only for a clear gain
      if (cost == 0 || (lc == best.lc ? c <= cost : c < 0.9 * cost)) {
        cost = c;
        best = {lc, r};
      }
    }
  }
  return best;
}

// k_vjp_gather: 128 columns per CTA, the rows strided over grid.y.
inline dim3 gather_grid(const Geom& g) {
  return dim3((unsigned)((g.pitch + 127) / 128), (unsigned)std::min<long long>(g.plane / g.pitch, 65535));
}

inline unsigned grid_for(long long n, int threads) {
  long long b = (n + threads - 1) / threads;
  if (b < 1) b = 1;
  if (b > 65535LL * 32) b = 65535LL * 32;
  return (unsigned)b;
}

long long n_interfaces(int nx, int nz, int dir) {
  return dir == MW_DIR_X ? (long long)nz * (nx + 1) : (long long)(nz + 1) * nx;
}

// Doubles of the workspace before the IEEE row table: the native form's
// interface adjoints of either direction (8 values per interface; one size
// serves every mode, and the IEEE form leaves them alone).
long long ieee_rows_off(int nx, int nz) {
  return 8 * std::max(n_interfaces(nx, nz, MW_DIR_X), n_interfaces(nx, nz, MW_DIR_Z));
}

}  // namespace

#if MW_CHECK
MW_OOB_COUNTER(oob_count_adjoint)
#endif

// mw_adjoint_split.cu
int launch_vjp_row_table(int nx, int nz, const double* hyc, const double* hytc, const double* hyi, const double* hyti,
                         const double* hypi, void* workspace, cudaStream_t stream);
int launch_vjp_split(int nx, int nz, double dx, double dz, double dt_full, const double* hyc, const void* table,
                     const double* forcing, const double* g_out, const double* g_base_a, const double* g_base_b,
                     int add_g_out, double* g_dst, double dt_stage, int direction, bool follows, cudaStream_t stream);
size_t vjp_split_table_bytes(int nz);

}  // namespace mw

using namespace mw;

extern "C" size_t mw_dirstage_vjp_workspace_bytes(int nx, int nz) {
  if (nx < 1 || nz < 1) return 0;
  const size_t ieee = sizeof(double) * (size_t)ieee_rows_off(nx, nz) + sizeof(RowV) * (size_t)(2 * nz + 5);
  return std::max(ieee, vjp_split_table_bytes(nz));
}

// Checks and launches one stage VJP; split mode expects the background table
// (launch_vjp_row_table) in the workspace when table_ready, else writes it.
static int vjp_stage(int nx, int nz, double dx, double dz, double dt_full, const double* hyc, const double* hytc,
                     const double* hyi, const double* hyti, const double* hypi, const double* forcing,
                     const double* g_out, const double* g_base_a, const double* g_base_b, int add_g_out,
                     double* g_dst, double dt_stage, int direction, int f64_mode, bool table_ready, bool follows,
                     void* workspace, size_t workspace_bytes, void* stream) {
  int st = check_grid(nx, nz);
  if (st) return st;
  MW_REQUIRE(finite_pos(dx) && finite_pos(dz) && finite_pos(dt_full), MW_ERR_INVALID_ARG,
             "dx, dz, dt_full must be finite and positive");
  MW_REQUIRE(std::isfinite(dt_stage), MW_ERR_INVALID_ARG, "dt_stage must be finite");
  MW_REQUIRE(direction == MW_DIR_X || direction == MW_DIR_Z, MW_ERR_INVALID_ARG, "direction must be 0 or 1");
  MW_REQUIRE(hyc && hytc && hyi && hyti && hypi && forcing && g_out && g_dst && workspace, MW_ERR_INVALID_ARG,
             "NULL pointer argument");
  MW_REQUIRE(aligned(forcing) && aligned(g_out) && aligned(g_dst) && ((uintptr_t)workspace % 8) == 0, MW_ERR_ALIGN,
             "misaligned pointer");
  const size_t bytes = sizeof(double) * 4 * (size_t)make_geom(nx, nz).plane;
  MW_REQUIRE(!ranges_overlap(g_dst, bytes, g_out, bytes), MW_ERR_ALIAS, "g_dst must not overlap g_out");
  MW_REQUIRE(!ranges_overlap(g_dst, bytes, forcing, bytes), MW_ERR_ALIAS, "g_dst must not overlap forcing");
  MW_REQUIRE((!g_base_a || g_base_a == g_dst || !ranges_overlap(g_dst, bytes, g_base_a, bytes)) &&
                 (!g_base_b || g_base_b == g_dst || !ranges_overlap(g_dst, bytes, g_base_b, bytes)),
             MW_ERR_ALIAS, "a base array must equal g_dst or not overlap it");
  MW_REQUIRE(valid_f64_mode(f64_mode), MW_ERR_INVALID_ARG, "f64_mode must be MW_F64_NATIVE, _SPLIT or _IEEE");
  const size_t need = mw_dirstage_vjp_workspace_bytes(nx, nz);
  MW_REQUIRE(workspace_bytes >= need, MW_ERR_WORKSPACE, "vjp workspace needs %zu bytes, got %zu", need,
             workspace_bytes);
  if (f64_mode == MW_F64_SPLIT) {
    if (!table_ready && (st = launch_vjp_row_table(nx, nz, hyc, hytc, hyi, hyti, hypi, workspace, (cudaStream_t)stream)))
      return st;
    return launch_vjp_split(nx, nz, dx, dz, dt_full, hyc, workspace, forcing, g_out, g_base_a, g_base_b, add_g_out,
                            g_dst, dt_stage, direction, follows || !table_ready, (cudaStream_t)stream);
  }
  const Geom g = make_geom(nx, nz);
  VjpArgs a;
  a.nx = nx;
  a.nz = nz;
  a.pitch = g.pitch;
  a.plane = g.plane;
  a.d = direction == MW_DIR_X ? dx : dz;
  a.hv = -kHvBeta * a.d / (16 * dt_full);
  a.dt_stage = dt_stage;
  a.hyc = hyc;
  a.hytc = hytc;
  a.hyi = hyi;
  a.hyti = hyti;
  a.hypi = hypi;
  a.forcing = forcing;
  a.gout = g_out;
  a.base_a = g_base_a;
  a.base_b = g_base_b;
  a.add_gout = add_g_out;
  a.gdst = g_dst;
  a.ws = (double*)workspace;
  a.nif = n_interfaces(nx, nz, direction);
  const bool ieee = f64_mode == MW_F64_IEEE;
  a.kc = dt_stage / a.d;
  a.ke = -a.hv * a.kc;
  cudaStream_t s = (cudaStream_t)stream;
  RowV* rows = (RowV*)((double*)workspace + ieee_rows_off(nx, nz));
  // Every launch of the call but its first may come in while the one before it ends (each waits before it touches
  // anything); `follows`: a launch of the same call came before this stage.
  if (ieee && !table_ready) {
    st = launch_overlapping(k_vjp_rows_ieee, dim3(grid_for(2 * nz + 5, 128)), 128, 0, s, false, "vjp row table", nz, hyc,
                            hytc, hyi, hyti, hypi, rows);
    if (st) return st;
    follows = true;
  }
  if (ieee && direction == MW_DIR_X) {  // one fused launch, a grid of resident CTAs at most
    int per_sm = 0, sms = 0, dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_vjp_ieee_x, kFXThreads, 0);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return fail(MW_ERR_CUDA, "vjp occupancy query: %s", cudaGetErrorString(e));
    const long long resident = (long long)std::max(1, per_sm) * sms;
    const int nseg = (nx + kFVCells - 1) / kFVCells;
    const long long total = (long long)nseg * nz;
    const long long grid = std::max(1LL, std::min(resident, (total + kFXWarps - 1) / kFXWarps));
    return launch_overlapping(k_vjp_ieee_x, dim3((unsigned)grid), kFXThreads, 0, s, follows, "vjp", a, rows, nseg, total);
  }
  if (ieee) {
    int sms = 0, dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const FzTile t = fz_tile(nx, nz, sms);
    const auto kern = t.lc == 5   ? k_vjp_ieee_z<5>
                      : t.lc == 7 ? k_vjp_ieee_z<7>
                      : t.lc == 6 ? k_vjp_ieee_z<6>
                      : t.lc == 4 ? k_vjp_ieee_z<4>
                      : t.lc == 3 ? k_vjp_ieee_z<3>
                      : t.lc == 2 ? k_vjp_ieee_z<2>
                                  : k_vjp_ieee_z<1>;
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, fz_smem(fz_max_rows(t.lc), t.lc));
    if (e != cudaSuccess) return fail(MW_ERR_CUDA, "vjp setup: %s", cudaGetErrorString(e));
    const long long tiles = (long long)((nx + (1 << t.lc) - 1) >> t.lc) * ((nz + t.rows - 1) / t.rows);
    return launch_overlapping(kern, dim3((unsigned)std::min(tiles, 1LL << 30)), kFZThreads, fz_smem(t.rows, t.lc), s,
                              follows, "vjp", a, rows, t.rows);
  }
  st = launch_overlapping(direction == MW_DIR_X ? k_vjp_iface<MW_DIR_X> : k_vjp_iface<MW_DIR_Z>,
                          dim3(grid_for(a.nif, 128)), 128, 0, s, follows, "vjp interface", a);
  if (st) return st;
  return launch_overlapping(direction == MW_DIR_X ? k_vjp_gather<MW_DIR_X> : k_vjp_gather<MW_DIR_Z>, gather_grid(g), 128,
                            0, s, true, "vjp gather", a);
}

extern "C" int mw_dirstage_vjp_f64(int nx, int nz, double dx, double dz, double dt_full, const double* hyc,
                                   const double* hytc, const double* hyi, const double* hyti, const double* hypi,
                                   const double* forcing, const double* g_out, const double* g_base_a,
                                   const double* g_base_b, int add_g_out, double* g_dst, double dt_stage,
                                   int direction, int f64_mode, void* workspace, size_t workspace_bytes,
                                   void* stream) {
  return vjp_stage(nx, nz, dx, dz, dt_full, hyc, hytc, hyi, hyti, hypi, forcing, g_out, g_base_a, g_base_b, add_g_out,
                   g_dst, dt_stage, direction, f64_mode, false, false, workspace, workspace_bytes, stream);
}

// ---------------------------------------------------------------------------
// Adjoint of one recorded time step (stages from mw_step_record_f64).  Per
// direction, in reverse (RK3 of solve/step.py:112-141):
//   s2bar = VJP(s2; g),  s1bar = VJP(s1; s2bar),  Sbar = g + s2bar + s1bar + VJP(S; s1bar).
extern "C" int mw_step_vjp_f64(int nx, int nz, double dx, double dz, double dt_full, double dt, const double* hyc,
                               const double* hytc, const double* hyi, const double* hyti, const double* hypi,
                               const double* stages, const double* g_out, double* g_in, double* gbuf, int reverse,
                               int f64_mode, void* workspace, size_t workspace_bytes, void* stream) {
  MW_REQUIRE(stages && g_out && g_in && gbuf, MW_ERR_INVALID_ARG, "NULL pointer argument");
  MW_REQUIRE(finite_pos(dt), MW_ERR_INVALID_ARG, "dt must be finite and positive");
  const size_t n = 4 * (size_t)make_geom(nx, nz).plane;
  MW_REQUIRE(!ranges_overlap(gbuf, 3 * n * sizeof(double), g_in, n * sizeof(double)) &&
                 !ranges_overlap(gbuf, 3 * n * sizeof(double), g_out, n * sizeof(double)),
             MW_ERR_ALIAS, "gbuf must not overlap g_in or g_out");
  double* gA = gbuf;
  double* gB = gbuf + n;
  double* gC = gbuf + 2 * n;
  const int dirs[2] = {reverse ? MW_DIR_X : MW_DIR_Z, reverse ? MW_DIR_Z : MW_DIR_X};
  const double* cur = g_out;
  int st;
  bool ready = false;  // a stage came before: the background table (split / IEEE modes) is written by the first
  for (int d = 1; d >= 0; --d) {
    const double* S = stages + (3 * d) * n;
    const double* s1 = S + n;
    const double* s2 = S + 2 * n;
    double* out = d == 1 ? gC : g_in;
    if ((st = vjp_stage(nx, nz, dx, dz, dt_full, hyc, hytc, hyi, hyti, hypi, s2, cur, nullptr, nullptr, 0, gA, dt,
                        dirs[d], f64_mode, ready, ready, workspace, workspace_bytes, stream)))
      return st;
    ready = true;
    if ((st = vjp_stage(nx, nz, dx, dz, dt_full, hyc, hytc, hyi, hyti, hypi, s1, gA, nullptr, nullptr, 0, gB, dt / 2,
                        dirs[d], f64_mode, ready, ready, workspace, workspace_bytes, stream)))
      return st;
    if ((st = vjp_stage(nx, nz, dx, dz, dt_full, hyc, hytc, hyi, hyti, hypi, S, gB, cur, gA, 1, out, dt / 3, dirs[d],
                        f64_mode, ready, ready, workspace, workspace_bytes, stream)))
      return st;
    cur = out;
  }
  return MW_OK;
}
