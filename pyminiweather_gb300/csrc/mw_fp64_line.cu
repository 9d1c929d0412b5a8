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
// cycles, however many of its lanes are active, and a stage is a chain of ~42
// of them.  On a small grid the stage kernels (mw_fp64_stage.cu) therefore pay
// for every row a thread marches and for the row tables a CTA forms: 30 us a z
// stage and 18 us an x stage at 100 x 50.  Here a cell is one lane's work: the
// cells of a line are cut into runs of at most 32 SL - 2, a warp per run (slots
// as in the x pass of mw_fp64_stage.cu), spread so that the SM partitions get
// equal numbers of warps, and the constants of an interface's row live in the
// registers of the lane that needs them (z) or are formed once per line (x).
#include <algorithm>
#include <atomic>

#include "mw_common.cuh"
#include "mw_fp64_flux.cuh"
#include "mw_fp64_line.cuh"

namespace mw {
namespace ieee {

// Most warps per CTA with SL slots per lane (as their registers allow).
__host__ __device__ constexpr int line_warps(int sl) { return sl == 1 ? 20 : 16; }
constexpr int kLineMax = 8;            // most lines per CTA
constexpr size_t kLineSmem = 200 << 10;

struct LineParams {
  LineArgs a;
  int n, nlines;         // cells per line, lines
  int log_lines, runs;   // lines per CTA (a power of two), runs per line
  int run;               // cells per run
  int lp;                // shared-memory pitch of a line
  int pitch;
  long long plane;
  double HV, IHV;        // HV = -12 hv of the direction and 1 / HV
  double c[3], dt[3];    // per stage HV dt_stage / (12 d) and dt_stage
  bool wait;             // launched while the kernel before it may still run
};

#define MW_LG(p, off) MW_AT((p), (off), 4 * P.plane)

// Line l of variable q in one of the two buffers, cell c at [c + 2].
__device__ __forceinline__ double* line_at(const LineParams& P, double* buf, int q, int l) {
  return buf + ((size_t)(q << P.log_lines) + l) * P.lp;
}

// Stores cell c of a line and, where it is a source of them, its halo images:
// periodic in x (ics/bcs.py:35-39), walls in z (bcs.py:92-148; hr[h] is
// hyc(halo row) / hyc(wall row) for rows -2, -1, nz, nz + 1).
template <int DIR>
__device__ __forceinline__ void put(double* line, int q, int c, int n, double v, const double* hr) {
  line[c + kHs] = v;
  if (DIR == MW_DIR_X) {
    if (c < kHs) line[n + kHs + c] = v;
    if (c >= n - kHs) line[c - n + kHs] = v;
  } else {
    if (c == 0)
      for (int h = 0; h < 2; ++h) line[h] = q == WMOM ? 0.0 : (q == UMOM ? v * hr[h] : v);
    if (c == n - 1)
      for (int h = 0; h < 2; ++h) line[n + kHs + h] = q == WMOM ? 0.0 : (q == UMOM ? v * hr[2 + h] : v);
  }
}

// The halo cells that cell c of a line is the source of, in a global array.
template <int DIR>
__device__ __forceinline__ void halo_out(const LineParams& P, double* g, int line, int c, const double v[4],
                                         const double* hr) {
  const int n = P.n;
  if (DIR == MW_DIR_X) {
    const long long row = (long long)(line + kHs) * P.pitch;
    for (int q = 0; q < 4; ++q) {
      if (c < kHs) MW_LG(g, q * P.plane + row + n + kHs + c) = v[q];
      if (c >= n - kHs) MW_LG(g, q * P.plane + row + c - n + kHs) = v[q];
    }
  } else {
    for (int q = 0; q < 4; ++q)
      for (int h = 0; h < 4; ++h)
        if (c == (h < 2 ? 0 : n - 1))
          MW_LG(g, q * P.plane + (long long)(h < 2 ? h : n + h) * P.pitch + line) =
              q == WMOM ? 0.0 : (q == UMOM ? v[q] * hr[h] : v[q]);
  }
}

// The CTA's lines between a global array and shared memory.  x: a warp per
// line and variable; z: consecutive threads take the CTA's columns of a row.
template <int DIR, typename Fn>
__device__ __forceinline__ void each_cell(const LineParams& P, int l0, int nl, Fn fn) {
  if (DIR == MW_DIR_X) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int ql = w; ql < 4 * nl; ql += nw) {
      const int q = ql / nl, l = ql - q * nl;
      const long long o = q * P.plane + (long long)(l0 + l + kHs) * P.pitch + kHs;
      for (int c = lane; c < P.n; c += 32) fn(q, l, c, o + c);
    }
  } else {
    for (int q = 0; q < 4; ++q)
      for (int i = threadIdx.x; i < (P.n << P.log_lines); i += blockDim.x) {
        const int l = i & ((1 << P.log_lines) - 1), c = i >> P.log_lines;
        if (l < nl) fn(q, l, c, q * P.plane + (long long)(c + kHs) * P.pitch + l0 + l + kHs);
      }
  }
}

template <int DIR, int SL>
__global__ void __launch_bounds__(line_warps(SL) * 32, 1) k_line_ieee(const __grid_constant__ LineParams P) {
  constexpr unsigned kAll = 0xffffffffu;
  extern __shared__ __align__(16) unsigned char smem_line[];
  __shared__ RowD rows[kLineMax];
  __shared__ double hr[4];
  const LineArgs& a = P.a;
  const int n = P.n, nl_cta = 1 << P.log_lines;
  double* buf[2] = {reinterpret_cast<double*>(smem_line),
                    reinterpret_cast<double*>(smem_line) + (size_t)4 * nl_cta * P.lp};
  const int l0 = blockIdx.x << P.log_lines, nl = min(nl_cta, P.nlines - l0);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int l = w / P.runs, rn = w - l * P.runs;   // the warp's line and run
  const bool live = l < nl;
  const int c0 = rn * P.run, c1 = live ? min(c0 + P.run, n) : 0;

  // row constants and wall ratios (backgrounds only: the kernel before it does not write them)
  RowD rz[SL];
  if (DIR == MW_DIR_X) {
    if (threadIdx.x < nl) {
      const int k = l0 + threadIdx.x + kHs;
      const double rt = MW_AT(a.hytc, k, P.nlines + 2 * kHs);
      rows[threadIdx.x] = row_consts(MW_AT(a.hyc, k, P.nlines + 2 * kHs), rt, kC0 * pow(rt, kGamma), P.HV, P.IHV);
    }
  } else {
    if (threadIdx.x < 4) {
      const int h = threadIdx.x < 2 ? threadIdx.x : n + threadIdx.x, src = threadIdx.x < 2 ? kHs : n + kHs - 1;
      hr[threadIdx.x] = MW_AT(a.hyc, h, n + 2 * kHs) / MW_AT(a.hyc, src, n + 2 * kHs);
    }
#pragma unroll
    for (int j = 0; j < SL; ++j) {
      const int i = min(max(c0 - 1 + 32 * j + lane, 0), n);
      const double rt12 = 12.0 * MW_AT(a.hyti, i, n + 1);
      rz[j].R = MW_AT(a.hyi, i, n + 1) * (12.0 * P.HV);
      rz[j].RT12 = rt12;
      rz[j].IRT12 = rcp(rt12, kAll);
      rz[j].P = MW_AT(a.hypi, i, n + 1) * (12.0 * P.IHV);
      rz[j].PC1 = rz[j].P * c_pow_g.c[1] * rz[j].IRT12;
    }
  }
  if (P.wait) asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (DIR == MW_DIR_Z) __syncthreads();  // hr
  each_cell<DIR>(P, l0, nl, [&](int q, int ll, int c, long long o) {
    put<DIR>(line_at(P, buf[0], q, ll), q, c, n, MW_LG(a.in, o), hr);
  });
  // the four x-halo columns of the wall halo rows, from the halo columns' own first and last rows
  if (DIR == MW_DIR_Z && blockIdx.x == 0 && threadIdx.x < 8) {
    double* g = threadIdx.x < 4 ? a.halo_in : a.halo_tmp;
    const int col = (threadIdx.x & 2) ? P.nlines + (threadIdx.x & 3) : (threadIdx.x & 1);
    if (g)
      for (int e = 0; e < 2; ++e) {
        double v[4];
        for (int q = 0; q < 4; ++q) v[q] = MW_LG(g, q * P.plane + (long long)(e ? n + kHs - 1 : kHs) * P.pitch + col);
        for (int q = 0; q < 4; ++q)
          for (int h = 2 * e; h < 2 * e + 2; ++h)
            MW_LG(g, q * P.plane + (long long)(h < 2 ? h : n + h) * P.pitch + col) =
                q == WMOM ? 0.0 : (q == UMOM ? v[q] * hr[h] : v[q]);
      }
  }
  double sw[SL];
#pragma unroll
  for (int j = 0; j < SL; ++j) {
    const int c = c0 - 2 + 32 * j + lane;  // the cell this slot updates
    sw[j] = 0.0;
    if (a.srcw && c >= c0 && c < c1) {
      const long long o = DIR == MW_DIR_X ? (long long)(l0 + l) * n + c : (long long)c * P.nlines + l0 + l;
      sw[j] = MW_AT(a.srcw, o, (long long)n * P.nlines);
    }
  }
  __syncthreads();

  double sv[SL][4];  // the direction's initial state at the updated cells
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    double* src = buf[s & 1];
    double* dst = buf[(s + 1) & 1];
    if (live) {
      double A[SL][4], D[SL][4], F[SL][4], wgt[SL];
      const int prev = (lane + 31) & 31;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double* ln = line_at(P, src, q, l) + kHs;
        double e[SL], qv[SL];
#pragma unroll
        for (int j = 0; j < SL; ++j) {
          const int i = min(c0 - 1 + 32 * j + lane, n);
          const double sm = ln[i - 1];
          cell_eq(sm, ln[i], ln[i + 1], e[j], qv[j]);
          if (s == 0) sv[j][q] = sm;
          if (q == DENS) wgt[j] = sm;
        }
#pragma unroll
        for (int j = 0; j < SL; ++j) {
          // slot j - 1's: lane 31 hands its slot of the group before to lane 0; slot 0 has none (not used)
          const double ep = __shfl_sync(kAll, j > 0 && lane == 31 ? e[j > 0 ? j - 1 : 0] : e[j], prev);
          const double qp = __shfl_sync(kAll, j > 0 && lane == 31 ? qv[j > 0 ? j - 1 : 0] : qv[j], prev);
          A[j][q] = qp + qv[j];
          D[j][q] = e[j] - ep;
        }
      }
#pragma unroll
      for (int j = 0; j < SL; ++j) {
        const int i = c0 - 1 + 32 * j + lane;
        if (DIR == MW_DIR_X)
          flux_x(A[j], D[j], rows[l], P.HV, P.IHV, kAll, F[j]);
        else
          flux_z(A[j], D[j], rz[j], P.HV, P.IHV, i <= 0 || i >= n, kAll, F[j]);
      }
#pragma unroll
      for (int j = 0; j < SL; ++j) {
        const int c = c0 - 2 + 32 * j + lane;
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const double Fp = __shfl_sync(kAll, j > 0 && lane == 31 ? F[j > 0 ? j - 1 : 0][q] : F[j][q], prev);
          v[q] = fma(P.c[s], Fp - F[j][q], sv[j][q]);
        }
        if (DIR == MW_DIR_Z) v[WMOM] = fma(-P.dt[s] * kGrav, wgt[j], v[WMOM]);
        if (a.srcw) v[WMOM] = fma(P.dt[s], sw[j], v[WMOM]);
        if (c >= c0 && c < c1) {
#pragma unroll
          for (int q = 0; q < 4; ++q) put<DIR>(line_at(P, dst, q, l), q, c, n, v[q], hr);
          const bool edge = DIR == MW_DIR_X ? (c < kHs || c >= n - kHs) : (c == 0 || c == n - 1);
          if (edge) {
            const int line = DIR == MW_DIR_X ? l0 + l : l0 + l + kHs;
            if (s == 0 && a.halo_in) halo_out<DIR>(P, a.halo_in, line, c, sv[j], hr);
            if (s == 1 && a.halo_tmp) halo_out<DIR>(P, a.halo_tmp, line, c, v, hr);
          }
        }
      }
    }
    __syncthreads();
    double* g = s == 0 ? a.s1 : (s == 1 ? a.s2 : a.out);
    if (g)
      each_cell<DIR>(P, l0, nl, [&](int q, int ll, int c, long long o) {
        MW_LG(g, o) = line_at(P, dst, q, ll)[c + kHs];
      });
  }
}

template <int DIR, int SL>
int launch_line_t(const LineParams& P, int ctas, int threads, size_t smem, cudaStream_t stream) {
  static std::atomic<int> done[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(MW_ERR_CUDA, "cudaGetDevice failed");
  if (dev < 0 || dev >= 64 || !done[dev].load(std::memory_order_relaxed)) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_line_ieee<DIR, SL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLineSmem);
    if (e != cudaSuccess) return fail(MW_ERR_CUDA, "line kernel shared memory: %s", cudaGetErrorString(e));
    if (dev >= 0 && dev < 64) done[dev].store(1, std::memory_order_relaxed);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)ctas);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = P.wait ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_line_ieee<DIR, SL>, P);
  if (e != cudaSuccess) return fail(MW_ERR_CUDA, "line kernel launch: %s", cudaGetErrorString(e));
  return MW_OK;
}

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

constexpr int run_cells(int sl) { return 32 * sl - 2; }

}  // namespace ieee

bool line_ieee_fits(int nx, int nz) {
  using namespace ieee;
  const int most = line_warps(2) * run_cells(2);
  return nx <= most && nz <= most && (long long)nx * nz <= kLineCellsMax;
}

int launch_line_ieee(int nx, int nz, double dx, double dz, double dt_full, double dt, const LineArgs& a, int direction,
                     bool overlap, cudaStream_t stream) {
  using namespace ieee;
  LineParams P;
  P.a = a;
  const bool isx = direction == MW_DIR_X;
  const Geom g = make_geom(nx, nz);
  P.n = isx ? nx : nz;
  P.nlines = isx ? nz : nx;
  P.pitch = g.pitch;
  P.plane = g.plane;
  P.lp = (P.n + 2 * kHs) | 1;
  const double d = isx ? dx : dz;
  P.HV = ieee_hv(d, dt_full);
  P.IHV = 1.0 / P.HV;
  for (int s = 0; s < 3; ++s) {
    P.dt[s] = dt / (3 - s);
    P.c[s] = P.dt[s] / (12.0 * d) * P.HV;
  }
  P.wait = overlap;
  int sms = 0, st = line_sms(&sms);
  if (st) return st;
  // Slots per lane and lines per CTA: the SM partitions' share of warp slots
  // decides the time (every slot group costs its partition the same FP64
  // instructions); among equals, z takes more lines (whole sectors of a row).
  int best_sl = 0, best_log = 0;
  long long best = 0;
  for (int sl = 1; sl <= 2; ++sl) {
    const int runs = (P.n + run_cells(sl) - 1) / run_cells(sl);
    for (int lg = 0; (1 << lg) <= kLineMax; ++lg) {
      const int warps = runs << lg;
      if (warps > line_warps(sl) || ((size_t)P.lp * sizeof(double) * 8 << lg) > kLineSmem) break;
      const long long ctas = (P.nlines + (1 << lg) - 1) >> lg;
      const long long per_sm = (ctas + sms - 1) / sms;
      const long long cost = per_sm * ((warps + 3) / 4) * sl;
      if (best_sl == 0 || cost < best || (cost == best && !isx && sl == best_sl)) {
        best = cost;
        best_sl = sl;
        best_log = lg;
      }
    }
  }
  MW_REQUIRE(best_sl, MW_ERR_SHAPE, "lines of %d cells do not fit a CTA", P.n);
  P.log_lines = best_log;
  const int min_runs = (P.n + run_cells(best_sl) - 1) / run_cells(best_sl);
  P.run = (P.n + min_runs - 1) / min_runs;
  P.runs = (P.n + P.run - 1) / P.run;
  const int threads = 32 * (P.runs << best_log);
  const int ctas = (P.nlines + (1 << best_log) - 1) >> best_log;
  const size_t smem = (size_t)P.lp * sizeof(double) * 8 << best_log;
  if (isx) return best_sl == 1 ? launch_line_t<MW_DIR_X, 1>(P, ctas, threads, smem, stream)
                               : launch_line_t<MW_DIR_X, 2>(P, ctas, threads, smem, stream);
  return best_sl == 1 ? launch_line_t<MW_DIR_Z, 1>(P, ctas, threads, smem, stream)
                      : launch_line_t<MW_DIR_Z, 2>(P, ctas, threads, smem, stream);
}

#if MW_CHECK
MW_OOB_COUNTER(oob_count_ieee_line)
#endif

}  // namespace mw
