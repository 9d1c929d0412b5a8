// mw_fp64_stage.cu -- direction-stage kernels in IEEE FP64 arithmetic with
// the fewest FP64 operations (f64_mode MW_F64_IEEE): the FP64 form of
// discrete_step (pyminiweather/solve/step.py:21-82).
//
// Every floating-point operation on state values is an FP64 add, multiply or
// FMA (no FP32 arithmetic on them, no double-FP32 pairs).  On GB300 the FP64
// pipe retires 2 operations per clock per SM, so one FP64 warp-instruction
// occupies it for 16 SM clocks, in which the SM can issue 64 other
// warp-instructions: the kernels are bound by their FP64 operation count, and
// integer work (conversions, index arithmetic, table look-ups) is nearly free.
// Against the reference's formulas (one pow, three divides and ~50 operations
// per interface, interpolate.py:82-186) a cell-stage costs 37 + n FP64
// operations, n the degree of the pressure series (z: one more, gravity):
//   - quantities are carried scaled by 12 and the two stencils are formed from
//     second differences e and q of the cells, shared by the neighbouring
//     interfaces: 5 operations per variable (ieee::cell_eq);
//   - fluxes are carried divided by HV = -12 hv, so that the hyperviscosity
//     term is the third difference itself, added by the FMA that forms the
//     advective term: rho is scaled by HV (one FMA with the background), so
//     that u / HV comes out of the reciprocal at no cost;
//   - one reciprocal per interface, 2 FP64 operations (ieee::rcp);
//   - pressure enters as the perturbation P_row ((1 + delta)^gamma - 1),
//     delta = (rho theta)' / (rho theta)_bg, P_row = C0 (rho theta)_bg^gamma:
//     exactly the reference's p - hy_pressure_int in z (hy_pressure_int is
//     C0 hy_dens_theta_int^gamma, ics/initial.py:105); in x the row constant
//     cancels in the flux difference.  (1 + delta)^gamma - 1 is its binomial
//     series summed by Horner's rule to the degree n that |delta| needs for a
//     truncation below 2^-54 relative (one FMA in a region at rest, up to 15
//     terms for |delta| < 1/8), and expm1(gamma log1p(delta)) beyond; the
//     single-grid kernels evaluate it as a polynomial in 12 (rho theta)' with
//     per-row coefficients (RowP), n operations in all;
//   - the stage update is out = init + c (F(i) - F(i+1)), c = HV dt / (12 d):
//     2 operations per value.
//
// x pass: warps walk runs of a row in blocks of 64 cells with no CTA barrier,
// lane l holding cells j+l and j+32+l (two independent FP64 chains) staged in
// the warp's shared-memory slice; e, q and the flux of the cell before come
// from the neighbouring lane, or from the block before.  z pass: one thread
// per column marching a tile of rows, e, q and the flux of the row before kept
// in registers.  Halo cells are never read: the periodic-x and wall-z rules of
// ics/bcs.py are applied to the indices and values as they are loaded.  On
// single grids the result at a cell depends on its neighbourhood alone, not on
// how the grid is split over warps (the series' degree is chosen per lane); the
// ensembles' x pass and the line kernels (mw_fp64_line.cu) take one degree per
// warp, so the last bits of a cell there may follow the cells its warp holds.
// Every global access goes through MW_AT (bounds-checked in the debug library).
#include <algorithm>
#include <atomic>

#include "mw_common.cuh"
#include "mw_ensemble.cuh"
#include "mw_fp64_flux.cuh"
#include "mw_fp64_math.cuh"
#include "mw_pow.cuh"

namespace mw {
namespace ieee {

constexpr int kXT = 256;            // threads per x CTA
constexpr int kZT = 128;            // columns per z CTA
constexpr int kZTileMax = 64;       // rows per z CTA
constexpr int kXRunBlocksMax = 16;  // blocks of 64 cells per warp of the x pass

// ---- arguments -------------------------------------------------------------
struct Args {
  int nx, nz, pitch;
  long long plane;
  const double* hyc;
  const double* hytc;
  const double* hyi;
  const double* hyti;
  const double* hypi;
  const double* srcw;
  const double* init;
  double* forcing;
  double* out;
  unsigned flags;
  double HV;    // -12 hv, hv = -hv_beta d / (16 dt_full) (interpolate.py:101,149)
  double IHV;   // 1 / HV
  double H12;   // 12 HV
  double I12;   // 12 / HV
  double c;     // HV dt_stage / (12 d)
  double dt;    // dt_stage (source terms)
  double gdt;   // -dt_stage grav (z)
  int z_tile;
  int r0, r1;   // output rows [r0, r1)
};

__device__ __forceinline__ int wrap_x(int j, int nx) { return j < 0 ? j + nx : (j >= nx ? j - nx : j); }

#define MW_F(a, off) MW_AT((a).forcing, (off), 4 * (a).plane)

// Forcing value of variable q at interior row k in [-2, nz+1] of the
// halo-indexed column col, with the wall rule of ics/bcs.py:92-148 in the halo rows.
__device__ __forceinline__ double zval(const Args& a, int q, int k, int col) {
  if (k >= 0 && k < a.nz) return MW_F(a, q * a.plane + (long long)(k + kHs) * a.pitch + col);
  if (q == WMOM) return 0.0;
  const int src = k < 0 ? kHs : a.nz + kHs - 1;
  const double s = MW_F(a, q * a.plane + (long long)src * a.pitch + col);
  if (q == UMOM) return s / MW_AT(a.hyc, src, a.nz + 2 * kHs) * MW_AT(a.hyc, k + kHs, a.nz + 2 * kHs);
  return s;
}

// Wall halo rows of one column of the forcing array: -2, -1 (bottom) from
// row 0, nz and nz+1 (top) from row nz-1.
__device__ __forceinline__ void write_z_halo_column(const Args& a, int col, bool bottom, bool top) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (!(h == 0 ? bottom : top)) continue;
    const int r0 = h == 0 ? -2 : a.nz;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double v0 = zval(a, q, r0, col), v1 = zval(a, q, r0 + 1, col);
      MW_F(a, q * a.plane + (long long)(r0 + kHs) * a.pitch + col) = v0;
      MW_F(a, q * a.plane + (long long)(r0 + 1 + kHs) * a.pitch + col) = v1;
    }
  }
}

// ---- x ---------------------------------------------------------------------
// A row is cut into runs of equal length (the last one shorter), one warp per
// run.  The warp walks the run in blocks of 64 slots with no CTA barrier: slot
// j of block b holds cell i = c0 - 1 + 64 b + j (lane l has slots l and 32 + l,
// two independent FP64 chains), forms the cell's e and q, the flux at the
// interface i between cells i - 1 and i, and updates cell i - 1.  e, q and the
// flux of slot j - 1 come from the lane before, or for slot 0 from slot 63 of
// the block before, so a run of n cells takes n + 2 slots.  The values of the
// next block are loaded one block ahead.
constexpr int kWSlots = 64;         // slots per block
constexpr int kXWarps = kXT / 32;
constexpr int kXShortBlocks = 8;    // most blocks of a run of the kernel that leaves out empty halves
constexpr int kXRunsMax = 4;        // most runs per warp of that kernel
struct SmemXW {
  double sS[kXWarps][4][kWSlots + 2];  // [warp][variable][cell i0-1 .. i0+64], i0 the cell of slot 0
};
__host__ __device__ inline int run_blocks(int cells) { return (cells + 2 + kWSlots - 1) / kWSlots; }
inline int run_halves(int cells) { return (cells + 2 + kWSlots / 2 - 1) / (kWSlots / 2); }

// Walks runs [g0, g1) of the row-major list of runs of `len` cells (nrun per
// row); row_at(k) gives the constants of row k.  Every lane of the warp calls
// it; prologue() runs once, after the first block's loads are issued (so that
// their latency overlaps it), also when the range is empty (it may contain a
// CTA barrier).  sS is the warp's shared-memory slice.
// SHORT: a run's last block that ends within its first 32 slots leaves the
// others' operations out, for rows of a few blocks (48 members of 64 to 512
// columns, two steps: 2073 -> 2036 us).
template <bool SHORT, typename RowAt, typename Prologue>
__device__ __forceinline__ void x_warp_walk(const Args& a, int nrun, int len, long long g0, long long g1, RowAt row_at,
                                            bool halo, double (*sS)[kWSlots + 2], Prologue prologue) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  // values of the block of row k whose slot 0 is cell i0: cells i0-1+lane, i0+31+lane and (lanes 0, 1)
  // i0+63+lane; slots beyond the run hold valid values that nothing uses.  Plain loads: with launches that
  // overlap, the launch before may write the forcing while this kernel is already resident (no ld.global.nc).
  auto load = [&](int k, int i0, double v[3][4]) {
    const long long row = (long long)(k + kHs) * a.pitch;
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      if (j < 2 || lane < 2) {
        const long long col = wrap_x(min(i0 - 1 + 32 * j + lane, a.nx + 1), a.nx) + kHs;
#pragma unroll
        for (int q = 0; q < 4; ++q) v[j][q] = MW_F(a, q * a.plane + row + col);
      }
    }
  };
  int k = (int)(g0 / nrun), rn = (int)(g0 - (long long)k * nrun);  // the current run: its row and place in the row
  int c0 = rn * len, c1 = min(c0 + len, a.nx), b = 0;
  double v[3][4] = {};
  if (g0 < g1) load(k, c0 - 1, v);
  prologue();
  double ce[4], cq[4], cF[4];  // e, q and flux of slots 32 .. 63 of the block before
#pragma unroll
  for (int q = 0; q < 4; ++q) ce[q] = cq[q] = cF[q] = 0.0;
  for (long long g = g0; g < g1;) {
    const int i0 = c0 - 1 + kWSlots * b;
    const long long row = (long long)(k + kHs) * a.pitch;
    __syncwarp();  // the previous block's values are read
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (j < 2 || lane < 2)
#pragma unroll
        for (int q = 0; q < 4; ++q) sS[q][32 * j + lane] = v[j][q];
    if (halo && rn == 0 && b == 0 && lane < 4) {  // columns 0, 1 <- nx, nx+1; nx+2, nx+3 <- 2, 3 (ics/bcs.py:35-39)
      const int dst = lane < 2 ? lane : a.nx + lane, src = lane < 2 ? a.nx + lane : lane;
#pragma unroll
      for (int q = 0; q < 4; ++q) MW_F(a, q * a.plane + row + dst) = MW_F(a, q * a.plane + row + src);
    }
    // cells updated by this lane
    const int ca = i0 - 1 + lane, cb = ca + 32;
    const bool ua = ca >= c0 && ca < c1, ub = cb < c1;
    double iva[4], ivb[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (ua) iva[q] = MW_AT(a.init, q * a.plane + row + ca + kHs, 4 * a.plane);
      if (ub) ivb[q] = MW_AT(a.init, q * a.plane + row + cb + kHs, 4 * a.plane);
    }
    const bool first = b == 0, both = !SHORT || i0 + 31 < c1;
    const int kc = k;
    // the next block: of this run, of the row's next run, or of the next row's first run
    if (++b == run_blocks(c1 - c0)) {
      b = 0;
      ++g;
      if (++rn == nrun) {
        rn = 0;
        ++k;
      }
      c0 = rn * len;
      c1 = min(c0 + len, a.nx);
    }
    if (g < g1) load(k, c0 - 1 + kWSlots * b, v);
    __syncwarp();
    const auto& rc = row_at(kc);
    const int prev = (lane + 31) & 31;
    auto update = [&](int c, const double* Fp, const double* F, const double* iv) {
      double o[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) o[q] = fma(a.c, Fp[q] - F[q], iv[q]);
      if (a.srcw) o[WMOM] = fma(a.dt, MW_AT(a.srcw, (long long)kc * a.nx + c, (long long)a.nx * a.nz), o[WMOM]);
#pragma unroll
      for (int q = 0; q < 4; ++q) MW_AT(a.out, q * a.plane + row + c + kHs, 4 * a.plane) = o[q];
    };
    auto block = [&](auto b_too) {
      constexpr bool B = decltype(b_too)::value;
      double Aa[4], Da[4], Ab[4], Db[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        double ea, qa, eb, qb;
        cell_eq(sS[q][lane], sS[q][lane + 1], sS[q][lane + 2], ea, qa);
        if (B) cell_eq(sS[q][32 + lane], sS[q][33 + lane], sS[q][34 + lane], eb, qb);
        double ep = __shfl_sync(kAll, lane == 31 ? ce[q] : ea, prev);
        double qp = __shfl_sync(kAll, lane == 31 ? cq[q] : qa, prev);
        if (first && lane == 0) {  // no cell before the run's first: its flux is not used
          ep = ea;
          qp = qa;
        }
        Aa[q] = qp + qa;
        Da[q] = ea - ep;
        if (B) {
          Ab[q] = __shfl_sync(kAll, lane == 31 ? qa : qb, prev) + qb;
          Db[q] = eb - __shfl_sync(kAll, lane == 31 ? ea : eb, prev);
          ce[q] = eb;
          cq[q] = qb;
        }
      }
      double Fa[4], Fb[4];
      flux_x(Aa, Da, rc, a.HV, a.IHV, kAll, Fa);
      if (B) flux_x(Ab, Db, rc, a.HV, a.IHV, kAll, Fb);
      // the flux at interface i - 1: the lane before's
      double Fpa[4], Fpb[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        Fpa[q] = __shfl_sync(kAll, lane == 31 ? cF[q] : Fa[q], prev);
        if (B) {
          Fpb[q] = __shfl_sync(kAll, lane == 31 ? Fa[q] : Fb[q], prev);
          cF[q] = Fb[q];
        }
      }
      if (ua) update(ca, Fpa, Fa, iva);
      if (B && ub) update(cb, Fpb, Fb, ivb);
    };
    if (both)
      block(std::true_type{});
    else
      block(std::false_type{});
  }
}

#ifndef MW_IEEE_X_MIN_BLOCKS
#define MW_IEEE_X_MIN_BLOCKS 2
#endif
// Single grid: consecutive runs of rows [r0, r1), one per warp (SHORT: up to
// kXRunsMax); the row constants (an FP64 power per row) are tabled once per CTA
// while the warps' first loads are in flight.  SHORT (x_warp_walk): rows of up to
// kXShortBlocks blocks whose runs end in the first half of one (a stage, 66x9000:
// 123 us with the empty halves, 103).
template <bool SHORT>
__global__ void __launch_bounds__(kXT, MW_IEEE_X_MIN_BLOCKS) k_stage_x_ieee_w(Args a, int nrun, int len, int per_warp,
                                                                               long long g0, long long g1) {
  __shared__ SmemXW sm;
  __shared__ RowP rows[kXWarps * (SHORT ? kXRunsMax : 1)];
  __shared__ PowTables pow_tables;
  if (!SHORT) per_warp = 1;
  const long long b0 = g0 + (long long)blockIdx.x * kXWarps * per_warp, b1 = min(b0 + kXWarps * per_warp, g1);
  const int row0 = (int)(b0 / nrun), nrows = (int)((b1 - 1) / nrun) - row0 + 1;  // at most one per run
  const int w = threadIdx.x >> 5;
  auto table = [&]() {
    load_pow_tables(pow_tables);
    __syncthreads();
    for (int r = threadIdx.x; r < nrows; r += kXT) {
      const double rt = MW_AT(a.hytc, row0 + r + kHs, a.nz + 2 * kHs);
      rows[r] = row_consts_p(MW_AT(a.hyc, row0 + r + kHs, a.nz + 2 * kHs), rt, kC0 * pow_gamma(rt, pow_tables), a.H12,
                             a.I12);
    }
    __syncthreads();
  };
  // overlapped with the launch before, the table comes before the wait; else it is formed under the first loads
  const bool early = a.flags & kFlagOverlap;
  if (early) table();
  overlap_wait();
  x_warp_walk<SHORT>(a, nrun, len, min(b0 + w * per_warp, b1), min(b0 + (w + 1) * per_warp, b1),
                     [&](int k) -> const RowP& { return rows[k - row0]; }, a.flags & MW_FLAG_WRITE_HALO, sm.sS[w], [&]() {
                       if (!early) table();
                     });
}

// ---- z ---------------------------------------------------------------------
struct SmemZ {
  RowP row[kZTileMax + 1];
};

// Columns [cb*NC, cb*NC+NC), rows [z0, z1), z1 - z0 <= kZTileMax; every
// thread of the CTA calls it.  hbot / htop: write the bottom / top wall halo
// rows of these columns (cb == 0 also of the four x-halo columns).
template <int NC>
__device__ __forceinline__ void z_tile(const Args& a, int cb, int z0, int z1, bool hbot, bool htop, SmemZ& sm) {
  for (int rr = threadIdx.x; rr <= z1 - z0; rr += NC) {
    const int k = z0 + rr;
    sm.row[rr] = row_consts_p(MW_AT(a.hyi, k, a.nz + 1), MW_AT(a.hyti, k, a.nz + 1), MW_AT(a.hypi, k, a.nz + 1), a.H12,
                              a.I12);
  }
  __syncthreads();
  overlap_wait();
  const int c = cb * NC + threadIdx.x;  // interior column
  if ((hbot || htop) && cb == 0 && threadIdx.x < 4)
    write_z_halo_column(a, threadIdx.x < 2 ? threadIdx.x : a.nx + threadIdx.x, hbot, htop);
  const unsigned mask = __ballot_sync(0xffffffffu, c < a.nx);
  if (c < a.nx) {
    const int col = c + kHs;
    if (hbot || htop) write_z_halo_column(a, col, hbot, htop);
    // s(k), s(k+1) and the e, q of cell k, k the row of the flux Fp just formed
    double s0[4], s1[4], e[4], qv[4], nxt[4], A[4], D[4], Fp[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const double sm2 = zval(a, q, z0 - 2, col), sm1 = zval(a, q, z0 - 1, col);
      s0[q] = zval(a, q, z0, col);
      s1[q] = zval(a, q, z0 + 1, col);
      nxt[q] = zval(a, q, z0 + 2, col);
      double e0, q0;
      cell_eq(sm2, sm1, s0[q], e0, q0);
      cell_eq(sm1, s0[q], s1[q], e[q], qv[q]);
      A[q] = q0 + qv[q];
      D[q] = e[q] - e0;
    }
    flux_z(A, D, sm.row[0], a.HV, a.IHV, z0 == 0, mask, Fp);
    for (int k = z0; k < z1; ++k) {
      const long long o = (long long)(k + kHs) * a.pitch + col;
      double iv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) iv[q] = MW_AT(a.init, q * a.plane + o, 4 * a.plane);
      const double rho_k = s0[DENS];  // forcing rho' at cell k (interpolate.py:248-250)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        double en, qn;
        cell_eq(s0[q], s1[q], nxt[q], en, qn);  // cell k + 1
        A[q] = qv[q] + qn;
        D[q] = en - e[q];
        e[q] = en;
        qv[q] = qn;
        s0[q] = s1[q];
        s1[q] = nxt[q];
      }
      if (k + 1 < z1) {  // the row the next iteration needs, loaded one step ahead
#pragma unroll
        for (int q = 0; q < 4; ++q) nxt[q] = zval(a, q, k + 3, col);
      }
      double Fn[4];
      flux_z(A, D, sm.row[k + 1 - z0], a.HV, a.IHV, k + 1 == a.nz, mask, Fn);
      double v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = fma(a.c, Fp[q] - Fn[q], iv[q]);
      v[WMOM] = fma(a.gdt, rho_k, v[WMOM]);
      if (a.srcw) v[WMOM] = fma(a.dt, MW_AT(a.srcw, (long long)k * a.nx + c, (long long)a.nx * a.nz), v[WMOM]);
#pragma unroll
      for (int q = 0; q < 4; ++q) MW_AT(a.out, q * a.plane + o, 4 * a.plane) = v[q];
#pragma unroll
      for (int q = 0; q < 4; ++q) Fp[q] = Fn[q];
    }
  }
  __syncthreads();  // the row table is rewritten by the next tile
}

// Tiles of a.z_tile rows of [a.r0, a.r1), one per CTA row.
__global__ void __launch_bounds__(kZT) k_stage_z_ieee(Args a, int tile0) {
  __shared__ SmemZ sm;
  const int tile = tile0 + blockIdx.y;  // grid.y is capped at 65535: one launch per 65535 tiles
  const int z0 = a.r0 + tile * a.z_tile, z1 = min(z0 + a.z_tile, a.r1);
  const bool halo = a.flags & MW_FLAG_WRITE_HALO;
  z_tile<kZT>(a, blockIdx.x, z0, z1, halo && z0 == 0, halo && z1 == a.nz, sm);
}

// ---- ensembles -------------------------------------------------------------
// One persistent launch per direction-stage walks a work list over all members
// (x items: member rows; z items: member column-block tiles).  Each member's
// stage constants were formed on the host with the plan, exactly as
// launch_stage_ieee forms them for a single grid, and the x row constants
// come from a table the step call writes once (no FP64 pow per row).
__device__ __forceinline__ Args member_args(const EnsStage& es, int e) {
  const mw_ens_member m = MW_AT(es.members, e, es.n_members);
  Args a;
  a.nx = m.nx;
  a.nz = m.nz;
  a.pitch = m.nx + 2 * kHs;
  a.plane = (long long)(m.nz + 2 * kHs) * a.pitch;
  a.hyc = es.hyc + m.cell_off;
  a.hytc = es.hytc + m.cell_off;
  a.hyi = es.hyi + m.int_off;
  a.hyti = es.hyti + m.int_off;
  a.hypi = es.hypi + m.int_off;
  a.srcw = nullptr;
  a.init = es.init + m.state_off;
  a.forcing = es.forcing + m.state_off;
  a.out = es.out + m.state_off;
  a.flags = es.flags;
  const EnsMemberConsts& c = MW_AT(reinterpret_cast<const EnsMemberConsts*>(es.mconsts), mconsts_index(es, e),
                                   (long long)kEnsConstsPerMember * es.n_members);
  a.HV = c.HV;
  a.IHV = c.IHV;
  a.H12 = 12.0 * c.HV;
  a.I12 = 12.0 * c.IHV;
  a.c = c.c;
  a.dt = c.dt;
  a.gdt = -c.dt * kGrav;
  a.z_tile = es.z_tile;
  a.r0 = 0;
  a.r1 = m.nz;
  return a;
}

static_assert(sizeof(RowD) <= kEnsRowBytes, "row-constant table entry size");

// The members' HV differ, so the table holds the constants for HV = 1; a warp scales its row's.
__global__ void k_ens_row_table_ieee(const double* hyc, const double* hytc, long long n, RowD* table) {
  for (long long j = blockIdx.x * (long long)blockDim.x + threadIdx.x; j < n; j += (long long)gridDim.x * blockDim.x) {
    const double rt = MW_AT(hytc, j, n);
    MW_AT(table, j, n) = row_consts(MW_AT(hyc, j, n), rt, kC0 * pow(rt, kGamma), 12.0, 12.0);
  }
}

// x items are rows (member, row), one per warp: the warp walks the row as one run.
__global__ void __launch_bounds__(kXT, MW_IEEE_X_MIN_BLOCKS) k_ens_x_ieee(EnsStage es) {
  __shared__ SmemXW sm;
  const int w = threadIdx.x >> 5;
  for (unsigned it = ens_take_warp(es.cursor); it < (unsigned)es.n_items; it = ens_take_warp(es.cursor)) {
    const int2 item = MW_AT(es.items, it, es.n_items);  // (member, row)
    const Args a = member_args(es, item.x);
    RowD r = MW_AT(reinterpret_cast<const RowD*>(es.xrows),
                   MW_AT(es.members, item.x, es.n_members).cell_off + item.y + kHs, es.n_xrows);
    r.R *= a.HV;
    r.P *= a.IHV;
    r.PC1 *= a.IHV;
    x_warp_walk<true>(a, 1, a.nx, (long long)item.y, (long long)item.y + 1, [&](int) -> const RowD& { return r; },
                a.flags & MW_FLAG_WRITE_HALO, sm.sS[w], []() {});
  }
  ens_finish(es.cursor);
}

__global__ void __launch_bounds__(kEnsZCols) k_ens_z_ieee(EnsStage es) {
  __shared__ SmemZ sm;
  __shared__ unsigned slot[2];
  int parity = 0;
  for (unsigned it = ens_take_cta(es.cursor, slot, parity); it < (unsigned)(es.n_items * es.z_parts);
       it = ens_take_cta(es.cursor, slot, parity)) {
    const int2 item = MW_AT(es.items, it / es.z_parts, es.n_items);  // (member, column block + ncb * tile)
    const Args a = member_args(es, item.x);
    const int ncb = (a.nx + kEnsZCols - 1) / kEnsZCols;
    const int cb = item.y % ncb, tile = item.y / ncb;
    int z0, z1;
    ens_part_rows(es, tile, it % es.z_parts, a.nz, z0, z1);
    if (z0 >= z1) continue;
    const bool halo = a.flags & MW_FLAG_WRITE_HALO;
    z_tile<kEnsZCols>(a, cb, z0, z1, halo && z0 == 0, halo && z1 == a.nz, sm);
  }
  ens_finish(es.cursor);
}

// CTAs of k_stage_x_ieee_w (which 0) / k_stage_z_ieee (which 1) resident on
// the current device, cached per device.
int resident_ctas(int which, int* out) {
  static std::atomic<int> cache[2][64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(MW_ERR_CUDA, "cudaGetDevice failed");
  const bool cached = dev >= 0 && dev < 64;
  if (cached && (*out = cache[which][dev].load(std::memory_order_relaxed)) > 0) return MW_OK;
  int per_sm = 0, sms = 0;
  cudaError_t e = which == 0 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_stage_x_ieee_w<false>, kXT, 0)
                             : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_stage_z_ieee, kZT, 0);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return fail(MW_ERR_CUDA, "occupancy query: %s", cudaGetErrorString(e));
  *out = std::max(1, per_sm) * sms;
  if (cached) cache[which][dev].store(*out, std::memory_order_relaxed);
  return MW_OK;
}

}  // namespace ieee

int launch_ens_ieee(const EnsStage& es, int grid) {
  using namespace ieee;
  if (es.n_items == 0) return MW_OK;
  if (es.direction == MW_DIR_X)
    k_ens_x_ieee<<<grid, kXT, 0, es.stream>>>(es);
  else
    k_ens_z_ieee<<<grid, kEnsZCols, 0, es.stream>>>(es);
  return check_launch("ensemble IEEE-FP64 stage launch");
}

int ens_ieee_occupancy(int direction, int* blocks_per_sm) {
  using namespace ieee;
  cudaError_t e = direction == MW_DIR_X
                      ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_ens_x_ieee, kXT, 0)
                      : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_ens_z_ieee, kEnsZCols, 0);
  if (e != cudaSuccess) return fail(MW_ERR_CUDA, "occupancy query: %s", cudaGetErrorString(e));
  return MW_OK;
}

int launch_ens_ieee_rowtable(const double* hyc, const double* hytc, long long n, void* table, cudaStream_t stream) {
  using namespace ieee;
  if (n <= 0) return MW_OK;
  MW_REQUIRE(((uintptr_t)table % 16) == 0, MW_ERR_ALIGN, "row table misaligned");
  const long long blocks = std::min<long long>((n + 127) / 128, 4096);
  k_ens_row_table_ieee<<<(unsigned)blocks, 128, 0, stream>>>(hyc, hytc, n, (RowD*)table);
  return check_launch("ensemble row-table launch");
}

// One direction-stage in the IEEE-FP64 form over output rows [r0, r1) (the
// whole grid: 0, nz); arguments validated by the caller.
int launch_stage_ieee(int nx, int nz, double dx, double dz, double dt_full, const double* hyc, const double* hytc,
                      const double* hyi, const double* hyti, const double* hypi, const double* srcw,
                      const double* init, double* forcing, double* out, double dt_stage, int direction,
                      unsigned flags, int r0, int r1, cudaStream_t stream) {
  using namespace ieee;
  MW_REQUIRE(0 <= r0 && r0 < r1 && r1 <= nz, MW_ERR_INVALID_ARG, "row range [%d, %d) outside [0, %d)", r0, r1, nz);
  const Geom g = make_geom(nx, nz);
  Args a;
  a.nx = nx;
  a.nz = nz;
  a.pitch = g.pitch;
  a.plane = g.plane;
  a.hyc = hyc;
  a.hytc = hytc;
  a.hyi = hyi;
  a.hyti = hyti;
  a.hypi = hypi;
  a.srcw = srcw;
  a.init = init;
  a.forcing = forcing;
  a.out = out;
  a.flags = flags;
  const double d = direction == MW_DIR_X ? dx : dz;
  const IeeeScale sc = ieee_scale(d, dt_full, dt_stage);
  a.HV = sc.HV;
  a.IHV = sc.IHV;
  a.H12 = sc.H12;
  a.I12 = sc.I12;
  a.c = sc.c;
  a.dt = dt_stage;
  a.gdt = -dt_stage * kGrav;
  a.r0 = r0;
  a.r1 = r1;
  const int rows = r1 - r0;
  if (direction == MW_DIR_Z) {
    // rows per z CTA: at most kZTileMax and at least 8 (each tile re-reads 4
    // window rows), chosen so that the launch is a whole number of resident
    // waves or just under (CTAs cost about the same, so a partly filled last
    // wave would idle SMs; one wave for the bands of the host-buffer step)
    int resident = 0, st = resident_ctas(1, &resident);
    if (st) return st;
    const long long ncb = (nx + kZT - 1) / kZT;
    const long long waves = std::max(1LL, ((long long)rows * ncb + (long long)kZTileMax * resident - 1) /
                                              ((long long)kZTileMax * resident));
    const long long tiles = std::max(1LL, waves * resident / ncb);
    a.z_tile = (int)std::max(8LL, std::min<long long>(kZTileMax, (rows + tiles - 1) / tiles));
  } else {
    a.z_tile = kZTileMax;
  }
  if (direction == MW_DIR_X) {
    // Runs per row: a warp's time is its blocks (and about a third of one to
    // start a run), and an SM's partitions each take two warps of every CTA it
    // gets, so the row is cut where ceil(CTAs / SMs) x (blocks + 1/3) is least
    // -- at most kXRunBlocksMax blocks, which leaves a large grid several waves.
    // A last block's empty half counts only where it is not left out, or where
    // the launch is too small for its operations to matter.
    int resident = 0, st = resident_ctas(0, &resident);
    if (st) return st;
    const long long sms = std::max(1, resident / MW_IEEE_X_MIN_BLOCKS);
    int nrun = 1;
    double best = 0.0;
    const int least = (int)(((long long)nx + kXRunBlocksMax * kWSlots - 1) / (kXRunBlocksMax * kWSlots));
    const int most = (int)(((long long)nx + kWSlots - 3) / (kWSlots - 2));
    const bool shortable = run_blocks(nx) <= kXShortBlocks;
    for (int n = least; n <= most; n = n == most ? n + 1 : std::min(most, n + std::max(1, n / 32))) {
      const int cells = (nx + n - 1) / n;
      const long long ctas = ((long long)n * rows + kXWarps - 1) / kXWarps;
      const double blocks = shortable && ctas > 2 * sms ? run_halves(cells) / 2.0 : run_blocks(cells);
      const double cost = (double)((ctas + sms - 1) / sms) * (blocks + 1.0 / 3);
      if (best == 0.0 || cost < best) {
        best = cost;
        nrun = n;
      }
    }
    const int len = (nx + nrun - 1) / nrun;
    nrun = (nx + len - 1) / len;
    const long long g0 = (long long)r0 * nrun, g1 = (long long)r1 * nrun;
    const bool odd = shortable && run_halves(len) % 2 == 1;
    // Rows of half a block or less: the table of their constants takes about as long as their cells, and no longer for
    // 32 rows than for 8 (2x2000000, a stage: 8.7 ms, 5.8).
    const int per_warp = odd && run_halves(len) == 1
                             ? (int)std::min<long long>(kXRunsMax, std::max<long long>(1, (g1 - g0) / (kXWarps * resident)))
                             : 1;
    const long long grid = (g1 - g0 + kXWarps * per_warp - 1) / (kXWarps * per_warp);
    MW_REQUIRE(grid <= 0x7fffffffLL, MW_ERR_SHAPE, "grid too large for the x direction-stage launch");
    return launch_overlapping(odd ? k_stage_x_ieee_w<true> : k_stage_x_ieee_w<false>, dim3((unsigned)grid), kXT, 0,
                              stream, flags & kFlagOverlap, "x IEEE-FP64 direction-stage", a, nrun, len, per_warp, g0, g1);
  } else {
    const int ntiles = (rows + a.z_tile - 1) / a.z_tile;
    for (int t0 = 0; t0 < ntiles; t0 += 65535) {
      dim3 grid((nx + kZT - 1) / kZT, (unsigned)std::min(ntiles - t0, 65535));
      const int st = launch_overlapping(k_stage_z_ieee, grid, kZT, 0, stream, (flags & kFlagOverlap) && t0 == 0,
                                        "z IEEE-FP64 direction-stage", a, t0);
      if (st) return st;
    }
  }
  return MW_OK;
}

#if MW_CHECK
MW_OOB_COUNTER(oob_count_ieee_stage)
#endif

}  // namespace mw
