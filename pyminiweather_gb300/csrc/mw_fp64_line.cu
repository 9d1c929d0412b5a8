// mw_fp64_line.cu -- the three RK stages of one direction in one launch, for
// grids whose lines fit a CTA (IEEE-FP64 form).
//
// The scheme is split by direction, so within a direction a row (x) or a
// column (z) never needs its neighbours: a CTA holds whole lines in shared
// memory and takes them through the three stages with two barriers, the state
// updated in place in global memory (replaces six launches of a step by two:
// evolve, pyminiweather/solve/step.py:85-143).
//
// What bounds it: a warp's FP64 instruction occupies its SM partition for 64
// cycles, however many of its lanes are active, and a stage is a chain of ~45
// of them.  On a small grid the stage kernels (mw_fp64_stage.cu) therefore pay
// for every row a thread marches and for the row tables a CTA forms: 30 us a z
// stage and 18 us an x stage at 100 x 50.  Here a cell is one lane's work: the
// cells of a line are cut into runs of at most 32 SL - 2 (14 in half slots), a
// warp per run (slots as in the x pass of mw_fp64_stage.cu), spread so that the SM partitions get
// equal numbers of warps, and the constants of an interface's row live in the
// registers of the lane that needs them (z) or are formed once per line (x).
// Lines may be cut into pieces, each CTA computing four cells more on either
// side of its piece in the first stage and two in the second, where that evens
// out the CTAs per SM; the direction's result then goes to another array.
#include <algorithm>
#include <atomic>

#include "mw_common.cuh"
#include "mw_fp64_flux.cuh"
#include "mw_fp64_line.cuh"
#include "mw_line.cuh"
#include "mw_pow.cuh"

namespace mw {
namespace ieee {

// Most warps per CTA with SL slots per lane (as their registers allow).
__host__ __device__ constexpr int line_warps(int sl) { return sl == 0 ? 24 : (sl == 1 ? 20 : 16); }
struct LineParams : LineGeom {
  double HV, IHV;        // HV = -12 hv of the direction and 1 / HV (ieee_scale)
  double H12, I12;       // 12 of either
  double c[3], dt[3];    // per stage HV dt_stage / (12 d) and dt_stage
};

// Line l of variable q in one of the two buffers.
__device__ __forceinline__ double* line_at(const LineParams& P, double* buf, int q, int l) {
  return buf + ((size_t)(q << P.log_lines) + l) * P.lp;
}

// Stores cell c of a line (line[c]) and, where it is a source of them, its halo
// images: periodic in x where the CTA holds the whole line (ics/bcs.py:35-39;
// the pieces of a cut row hold their neighbours' cells instead), walls in z
// (bcs.py:92-148; hr[h] is hyc(halo row) / hyc(wall row) for rows -2, -1, nz,
// nz + 1).
template <int DIR>
__device__ __forceinline__ void put(double* line, int q, int c, int n, bool whole, double v, const double* hr) {
  line[c] = v;
  if (DIR == MW_DIR_X) {
    if (whole && c < kHs) line[n + c] = v;
    if (whole && c >= n - kHs) line[c - n] = v;
  } else {
    if (c == 0)
      for (int h = 0; h < 2; ++h) line[h - 2] = q == WMOM ? 0.0 : (q == UMOM ? v * hr[h] : v);
    if (c == n - 1)
      for (int h = 0; h < 2; ++h) line[n + h] = q == WMOM ? 0.0 : (q == UMOM ? v * hr[2 + h] : v);
  }
}

// flux_x or flux_z (mw_fp64_flux.cuh) by the two halves of a warp: A and D of (DENS, UMOM) in lanes 0 .. 15, of
// (WMOM, RHOT) of the same interfaces in lanes 16 .. 31, F likewise; the same operations on each value.
template <int DIR>
__device__ __forceinline__ void flux_halves(const double A[2], const double D[2], const RowD& r, double HV, double IHV,
                                            bool wall, double F[2]) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, lo = lane & 15, hi = lo | 16;
  const bool up = lane >= 16;
  const double AD = __shfl_sync(kAll, A[0], lo), AT = __shfl_sync(kAll, A[1], hi);
  double m = DIR == MW_DIR_X ? __shfl_sync(kAll, A[1], lo) : __shfl_sync(kAll, A[0], hi);  // the direction's momentum
  double d0 = D[0];
  if (DIR == MW_DIR_Z && wall) {
    m = 0.0;
    if (!up) d0 = 0.0;
  }
  const double u = m * rcp(fma(HV, AD, r.R), kAll);
  const double p = pressure(AT, r, DIR == MW_DIR_X ? D[1] : d0, kAll);
  const double t = AT + r.RT12;
  if (DIR == MW_DIR_X) {
    F[0] = fma(up ? u : IHV, up ? A[0] : m, d0);
    F[1] = fma(up ? t : m, u, up ? D[1] : p);
  } else {
    F[0] = fma(up ? u : IHV, m, up ? p : d0);
    F[1] = fma(u, up ? t : A[1], D[1]);
  }
}

// SL slots per lane; SL = 0: the lanes of a warp's two halves share sixteen slots, two variables each, which shortens
// a stage's chain of FP64 instructions (25 instead of 41) where a grid leaves SM partitions idle.
template <int DIR, int SL>
__global__ void __launch_bounds__(line_warps(SL) * 32, 1) k_line_ieee(const __grid_constant__ LineParams P) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int NS = SL == 0 ? 1 : SL, NV = SL == 0 ? 2 : 4;  // slots and variables of a lane
  extern __shared__ __align__(16) unsigned char smem_line[];
  __shared__ RowD rows[kLineMax];
  __shared__ double hr[4];
  __shared__ PowTables pow_tables;  // x
  const LineArgs& a = P.a;
  const int n = P.n, nl_cta = 1 << P.log_lines;
  const int group = blockIdx.x / P.pieces, pc = blockIdx.x - group * P.pieces;
  const int l0 = group << P.log_lines, nl = min(nl_cta, P.nlines - l0);
  const bool whole = P.pieces == 1;
  const int p0 = pc * P.piece, p1 = min(p0 + P.piece, n);  // the CTA's cells
  // first and last + 1 cell of a stage's result that the next stages need of this piece
  auto first = [&](int s) { return whole ? 0 : (DIR == MW_DIR_X ? p0 - 4 + 2 * s : max(p0 - 4 + 2 * s, 0)); };
  auto past = [&](int s) { return whole ? n : (DIR == MW_DIR_X ? p1 + 4 - 2 * s : min(p1 + 4 - 2 * s, n)); };
  // the two buffers, so that cell c of a line is at [c] from line_at
  double* buf[2] = {reinterpret_cast<double*>(smem_line) + (whole ? kHs : 6 - p0),
                    reinterpret_cast<double*>(smem_line) + (size_t)4 * nl_cta * P.lp + (whole ? kHs : 6 - p0)};
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int sub = SL == 0 ? lane & 15 : lane, q0 = SL == 0 ? (lane >> 4) * 2 : 0;  // the lane's slot and first variable
  const int l = w / P.runs, rn = w - l * P.runs;   // the warp's line and run
  const int c0 = first(0) + rn * P.run, c1 = min(c0 + P.run, past(0));
  const bool live = l < nl && c0 < c1;

  // row constants and wall ratios (backgrounds only: the kernel before it does not write them)
  RowD rz[NS];
  if (DIR == MW_DIR_X) {
    load_pow_tables(pow_tables);
    double r = 0.0, rt = 1.0;
    if (threadIdx.x < nl) {
      r = MW_AT(a.hyc, l0 + threadIdx.x + kHs, P.nlines + 2 * kHs);
      rt = MW_AT(a.hytc, l0 + threadIdx.x + kHs, P.nlines + 2 * kHs);
    }
    __syncthreads();
    if (w == 0) {
      const double pr = kC0 * pow_gamma(rt, pow_tables), irt = rcp(12.0 * rt, kAll), p = pr * P.I12;
      if (lane < nl) rows[lane] = {r * P.H12, 12.0 * rt, irt, p, p * c_pow_g.c[1] * irt};
    }
  } else {
    if (threadIdx.x < 4) {
      const int h = threadIdx.x < 2 ? threadIdx.x : n + threadIdx.x, src = threadIdx.x < 2 ? kHs : n + kHs - 1;
      hr[threadIdx.x] = MW_AT(a.hyc, h, n + 2 * kHs) / MW_AT(a.hyc, src, n + 2 * kHs);
    }
#pragma unroll
    for (int j = 0; j < NS; ++j) {
      const int i = min(max(c0 - 1 + 32 * j + sub, 0), n);
      const double rt12 = 12.0 * MW_AT(a.hyti, i, n + 1);
      rz[j].R = MW_AT(a.hyi, i, n + 1) * P.H12;
      rz[j].RT12 = rt12;
      rz[j].IRT12 = rcp(rt12, kAll);
      rz[j].P = MW_AT(a.hypi, i, n + 1) * P.I12;
      rz[j].PC1 = rz[j].P * c_pow_g.c[1] * rz[j].IRT12;
    }
  }
  overlap_wait();
  if (gridDim.x <= kLineFewCtas) overlap_next();
  if (DIR == MW_DIR_Z) __syncthreads();  // hr
  {
    const int ca = whole ? 0 : (DIR == MW_DIR_X ? p0 - 6 : max(p0 - 6, 0));
    const int cb = whole ? n : (DIR == MW_DIR_X ? p1 + 6 : min(p1 + 6, n));
    each_cell4<DIR>(P, l0, nl, ca, cb, [&](int ll, int c, long long o) {
      double v[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = MW_LG(a.in, q * P.plane + o);
#pragma unroll
      for (int q = 0; q < 4; ++q) put<DIR>(line_at(P, buf[0], q, ll), q, c, n, whole, v[q], hr);
    });
  }
  double sw[NS];
#pragma unroll
  for (int j = 0; j < NS; ++j) {
    int c = c0 - 2 + 32 * j + sub;  // the cell this slot updates
    sw[j] = 0.0;
    if (a.srcw && live && c >= c0 && c < c1) {
      if (DIR == MW_DIR_X) c = c < 0 ? c + n : (c >= n ? c - n : c);
      const long long o = DIR == MW_DIR_X ? (long long)(l0 + l) * n + c : (long long)c * P.nlines + l0 + l;
      sw[j] = MW_AT(a.srcw, o, (long long)n * P.nlines);
    }
  }
  __syncthreads();

  double sv[NS][NV];  // the direction's initial state at the updated cells
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    double* src = buf[s & 1];
    double* dst = buf[(s + 1) & 1];
    if (live) {
      double A[NS][NV], D[NS][NV], F[NS][NV], wgt[NS];
      const int prev = SL == 0 ? (lane & 16) | ((lane + 15) & 15) : (lane + 31) & 31;
#pragma unroll
      for (int q = 0; q < NV; ++q) {
        const double* ln = line_at(P, src, q0 + q, l);
        double e[NS], qv[NS];
#pragma unroll
        for (int j = 0; j < NS; ++j) {
          // slots beyond the stage's cells repeat its last ones (not used)
          const int i = min(max(c0 - 1 + 32 * j + sub, first(s) - 1), past(s));
          const double sm = ln[i - 1];
          cell_eq(sm, ln[i], ln[i + 1], e[j], qv[j]);
          if (s == 0) sv[j][q] = sm;
          if (q == DENS) wgt[j] = SL == 0 ? line_at(P, src, DENS, l)[i - 1] : sm;
        }
#pragma unroll
        for (int j = 0; j < NS; ++j) {
          // slot j - 1's: lane 31 hands its slot of the group before to lane 0; slot 0 has none (not used)
          const double ep = __shfl_sync(kAll, j > 0 && lane == 31 ? e[j > 0 ? j - 1 : 0] : e[j], prev);
          const double qp = __shfl_sync(kAll, j > 0 && lane == 31 ? qv[j > 0 ? j - 1 : 0] : qv[j], prev);
          A[j][q] = qp + qv[j];
          D[j][q] = e[j] - ep;
        }
      }
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        const int i = c0 - 1 + 32 * j + sub;
        if constexpr (SL == 0)
          flux_halves<DIR>(A[j], D[j], DIR == MW_DIR_X ? rows[l] : rz[j], P.HV, P.IHV, i <= 0 || i >= n, F[j]);
        else if (DIR == MW_DIR_X)
          flux_x(A[j], D[j], rows[l], P.HV, P.IHV, kAll, F[j]);
        else
          flux_z(A[j], D[j], rz[j], P.HV, P.IHV, i <= 0 || i >= n, kAll, F[j]);
      }
#pragma unroll
      for (int j = 0; j < NS; ++j) {
        const int c = c0 - 2 + 32 * j + sub;
        double v[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) {
          const double Fp = __shfl_sync(kAll, j > 0 && lane == 31 ? F[j > 0 ? j - 1 : 0][q] : F[j][q], prev);
          v[q] = fma(P.c[s], Fp - F[j][q], sv[j][q]);
        }
        // of a warp's lower half this is no variable: its values are left as they are
        double& vw = v[SL == 0 ? 0 : WMOM];
        const bool has_w = SL != 0 || q0 == WMOM;
        if (DIR == MW_DIR_Z) {
          const double g = fma(-P.dt[s] * kGrav, wgt[j], vw);
          vw = has_w ? g : vw;
        }
        if (a.srcw) {
          const double f = fma(P.dt[s], sw[j], vw);
          vw = has_w ? f : vw;
        }
        if (c >= max(c0, first(s)) && c < min(c1, past(s)) && (SL != 0 || sub >= 2)) {
#pragma unroll
          for (int q = 0; q < NV; ++q) put<DIR>(line_at(P, dst, q0 + q, l), q0 + q, c, n, whole, v[q], hr);
          const bool edge = c < p0 || c >= p1 ? false : DIR == MW_DIR_X ? (c < kHs || c >= n - kHs) : (c == 0 || c == n - 1);
          if (edge) {
            const int line = DIR == MW_DIR_X ? l0 + l : l0 + l + kHs;
            if (s == 0 && a.halo_in) halo_out<DIR, NV>(P, a.halo_in, line, c, sv[j], hr, q0);
            if (s == 1 && a.halo_tmp) halo_out<DIR, NV>(P, a.halo_tmp, line, c, v, hr, q0);
          }
        }
      }
    }
    __syncthreads();
    if (s == 2) overlap_next();  // at the latest (kLineFewCtas)
    double* g = s == 0 ? a.s1 : (s == 1 ? a.s2 : a.out);
    if (g)
      each_cell4<DIR>(P, l0, nl, p0, p1, [&](int ll, int c, long long o) {
#pragma unroll
        for (int q = 0; q < 4; ++q) MW_LG(g, q * P.plane + o) = line_at(P, dst, q, ll)[c];
      });
  }
  if (DIR == MW_DIR_Z && blockIdx.x == 0 && threadIdx.x < 8) halo_corners(P, hr);
}

template <int DIR, int SL>
int launch_line_t(const LineParams& P, int ctas, int threads, size_t smem, bool overlap, cudaStream_t stream) {
  static std::atomic<int> done[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(MW_ERR_CUDA, "cudaGetDevice failed");
  if (dev < 0 || dev >= 64 || !done[dev].load(std::memory_order_relaxed)) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_line_ieee<DIR, SL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLineSmem);
    if (e != cudaSuccess) return fail(MW_ERR_CUDA, "line kernel shared memory: %s", cudaGetErrorString(e));
    if (dev >= 0 && dev < 64) done[dev].store(1, std::memory_order_relaxed);
  }
  return launch_overlapping(k_line_ieee<DIR, SL>, dim3((unsigned)ctas), threads, smem, stream, overlap, "line kernel", P);
}

// two slots of a run repeat its neighbours' (x pass of mw_fp64_stage.cu)
constexpr LineKind kIeeeLines = {0, 2, {line_warps(0), line_warps(1), line_warps(2)}, {80, 96, 128}, 2, 64, 0, 0.0};

constexpr int kMaxPieces = 16, kMinPiece = 24;
// The last piece may be shorter than the others by a cell per piece; the halo slots beside it hold six cells.
static_assert(kMinPiece - (kMaxPieces - 1) > 6, "a last piece must be longer than its neighbours' halo");
// A warp of half slots against one of whole ones: 0.61 in FP64 instructions, more in time (us a step, eight a call:
// 60x30 20.5 -> 16.6, 100x50 20.0 -> 17.6; where partitions get two warps for one it loses, 200x100 31.0 -> 36.2 a step
// in calls of one).
constexpr double kHalfCost = 0.75;

// The spread with the least time.  An SM that gets m CTAs of W warps with SL
// slots per lane gives its four partitions m W SL / 4 slot groups each, every
// one the same FP64 instructions, and that is what the time follows: measured
// over every spread of thirteen grids from 100x50 to 900x300, both directions in
// turn, 5.5 to 6.5 us a group (401x199, x: whole rows in 14 warps, two CTAs on
// some SMs, 7 groups, 42 us; in three pieces of five warps, four CTAs, 5 groups,
// 30 us).  Where all CTAs of an SM are resident at once its fullest partition
// counts (nearly: m W / 4 rounded up); else m is rounded up to whole turns of
// the resident CTAs, but for a last turn that fewer than half would fill.  Two
// slots per lane with less than two warps per partition wait on their own
// latency.  The factors near 1 break ties: more resident CTAs (their heads and
// tails fill one another), fewer pieces, fewer CTAs, in z whole sectors.
//
// The double-FP32 form's warps hide one another's latency instead, and its time
// follows the warps of the SM with the most CTAs, partition by partition, and
// part of a CTA's own for its head and tail, less where more CTAs are resident
// to fill them.  CTAs of under four warps leave partitions idle, and single
// columns use a quarter of a sector.  Over every spread of eleven grids from
// 100x50 to 1250x799, both directions in turn, the rule takes one within 2 % of
// the fastest but for 300x150, x (4 %): 512x256, x: whole rows in 17 warps 46.7 us
// a step, five pieces of four warps 43.1; 880x620, z: twelve pieces of two columns
// in four warps 122 us, of one column in two warps 129, three in 14 warps 150.  The
// FP32 form takes the same rule (within 3 % of the fastest spread from 100x50 to
// 1000x1000).
LineSpread spread_lines(const LineKind& kind, int n, int nlines, bool isx, int sms) {
  LineSpread best;
  double least = 0.0;
  for (int sl = kind.min_slots; sl <= kind.max_slots; ++sl)
    for (int pieces = 1; pieces == 1 || (pieces <= kMaxPieces && (n + pieces - 1) / pieces >= kMinPiece); ++pieces) {
      const int piece = (n + pieces - 1) / pieces;
      if ((n + piece - 1) / piece != pieces) continue;  // an empty last piece
      const int range = pieces == 1 ? n : piece + 8;
      if (pieces > 1 && range >= n) break;
      const int cells = (sl == 0 ? 16 : 32 * sl) - kind.shared_slots, runs = (range + cells - 1) / cells;
      const int lp = (pieces == 1 ? n + 2 * kHs : piece + 12) | 1;
      for (int lg = 0; (1 << lg) <= kLineMax; ++lg) {
        const int warps = runs << lg;
        const size_t smem = line_smem(kind, lp, lg, isx);
        if (warps > kind.warps[sl] || smem > kLineSmem) break;
        const int resident = std::min((int)(65536 / (kind.regs[sl] * 32 * warps)), (int)((220 << 10) / smem));
        const double load = (double)((nlines + (1 << lg) - 1) >> lg) * pieces / sms;
        const double turns = std::min(std::ceil(load / resident) * resident, load + 0.5 * resident) * warps / 4.0;
        const double once = std::ceil(load) * warps / 4.0;
        double cost;
        if (kind.tail > 0.0) {
          cost = (once + kind.tail * std::max(warps, 4)) * (1.0 + 0.3 / resident) * (1.0 + 0.001 * pieces) *
                 (warps < 4 ? 1.1 : 1.0) * (!isx && lg == 0 ? 1.2 : 1.0);
        } else {
          cost = (sl == 0 ? kHalfCost : sl) * (load <= resident ? 0.1 * once + 0.9 * std::ceil(once) : turns);
          cost *= (1.0 + 0.1 / resident) * (1.0 + 0.001 * load) * (pieces > 1 ? 1.01 : 1.0) *
                  (!isx && lg == 0 ? 1.03 : 1.0) * (sl == 2 && once < 2.0 ? 1.3 : 1.0);
        }
        if (best.runs == 0 || cost < least) {
          least = cost;
          const int run = (range + runs - 1) / runs;
          best = {sl, lg, pieces, piece, (range + run - 1) / run, run, lp};
        }
      }
    }
  return best;
}

}  // namespace ieee

int line_sms(int* out) {
  static std::atomic<int> cache[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(MW_ERR_CUDA, "cudaGetDevice failed");
  const bool cached = dev >= 0 && dev < 64;
  if (cached && (*out = cache[dev].load(std::memory_order_relaxed)) > 0) return MW_OK;
  const cudaError_t e = cudaDeviceGetAttribute(out, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return fail(MW_ERR_CUDA, "device query: %s", cudaGetErrorString(e));
  if (cached) cache[dev].store(*out, std::memory_order_relaxed);
  return MW_OK;
}

LinePlan line_plan(const LineKind& kind, int nx, int nz, int sms) {
  LinePlan p;
  p.x = ieee::spread_lines(kind, nx, nz, true, sms);
  p.z = ieee::spread_lines(kind, nz, nx, false, sms);
  p.fits = p.x.runs > 0 && p.z.runs > 0;
  p.cut = p.x.pieces > 1 || p.z.pieces > 1;
  return p;
}

int line_ieee_plan(int nx, int nz, LinePlan* plan) {
  using namespace ieee;
  *plan = LinePlan();
  if ((long long)nx * nz > kLineCellsMax) return MW_OK;
  int sms = 0, st = line_sms(&sms);
  if (st) return st;
  *plan = line_plan(kIeeeLines, nx, nz, sms);
  return MW_OK;
}

int launch_line_ieee(const LinePlan& plan, int nx, int nz, double dx, double dz, double dt_full, double dt,
                     const LineArgs& a, int direction, bool overlap, cudaStream_t stream) {
  using namespace ieee;
  LineParams P;
  P.a = a;
  const bool isx = direction == MW_DIR_X;
  const double d = isx ? dx : dz;
  const IeeeScale sc = ieee_scale(d, dt_full, dt);
  P.HV = sc.HV;
  P.IHV = sc.IHV;
  P.H12 = sc.H12;
  P.I12 = sc.I12;
  for (int s = 0; s < 3; ++s) {
    P.dt[s] = dt / (3 - s);
    P.c[s] = sc.c / (3 - s);
  }
  const LineSpread& sp = isx ? plan.x : plan.z;
  MW_REQUIRE(sp.pieces == 1 || a.in != a.out, MW_ERR_ALIAS, "a direction of cut lines needs another array for its result");
  int ctas, threads;
  set_line_geom(&P, sp, nx, nz, isx, &ctas, &threads);
  const size_t smem = line_smem(kIeeeLines, P.lp, P.log_lines, isx);
  const auto launch = isx ? (sp.sl == 0   ? launch_line_t<MW_DIR_X, 0>
                             : sp.sl == 1 ? launch_line_t<MW_DIR_X, 1>
                                          : launch_line_t<MW_DIR_X, 2>)
                          : (sp.sl == 0   ? launch_line_t<MW_DIR_Z, 0>
                             : sp.sl == 1 ? launch_line_t<MW_DIR_Z, 1>
                                          : launch_line_t<MW_DIR_Z, 2>);
  return launch(P, ctas, threads, smem, overlap, stream);
}

#if MW_CHECK
MW_OOB_COUNTER(oob_count_ieee_line)
#endif

}  // namespace mw
