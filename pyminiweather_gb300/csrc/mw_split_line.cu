// mw_split_line.cu -- the three RK stages of one direction in one launch, for
// grids whose lines fit a CTA (double-FP32 form).
//
// As mw_fp64_line.cu (whole lines or pieces of lines in shared memory, a warp
// per run of a line, the launches of a call overlapping), with the arithmetic
// of mw_split_stage.cu value for value: the first stage's result stays a pair,
// as it does between the stage kernels of a step, the second's and third's are
// FP64 and the former is split again where the third reads it.  Shared memory
// holds, per cell, the forcing as pairs twice (a stage's input and its result)
// and four FP64 values on their way in or out (96 bytes).  A lane owns an
// interface of a run and the cell to its right; the initial state of that cell
// stays in its registers through the stages.
//
// What bounds it: the FP32 pipe, ~1000 cycles of an SM partition per warp and
// stage, once a few warps a partition hide its chain of dependent operations,
// and below that the chain itself.  A stage kernel of a small grid waits on its
// loads and row tables as well, six times a step: 63 us at 100 x 50, 13 here.
#include <algorithm>
#include <atomic>

#include "mw_common.cuh"
#include "mw_line.cuh"
#include "mw_pow.cuh"
#include "mw_split_flux.cuh"

namespace mw {
namespace {

constexpr int kSplitWarps = 20;  // most per CTA (88 registers a thread)
constexpr LineKind kSplitLines = {1, 1, {0, kSplitWarps, 0}, {0, 88, 0}, 1, 96, sizeof(RowS), 0.4};

struct SplitLineParams : LineGeom {
  dwc hv12, d12, gz12;   // 12 hv, 12 d, 12 dz grav
  dwc c12;               // of the first stage: dt_stage / (12 d)
  double c12s[3];        // per stage 2^896 dt_stage / (12 d)
};

// Stores the pairs p of cell c of a line (planes `pl` apart) and the halo cells it is the source of, by the rules of
// put in mw_fp64_line.cu; hr[h]: hyc(halo row) / hyc(wall row).  U(h): the momentum along x of halo row h as a pair.
template <int DIR, typename U>
__device__ __forceinline__ void put_pairs(dw2* line, size_t pl, int c, int n, bool whole, const dw2 p[2], U u_of) {
  line[c] = p[0];
  line[pl + c] = p[1];
  if (DIR == MW_DIR_X) {
    if (whole && c < kHs) {
      line[n + c] = p[0];
      line[pl + n + c] = p[1];
    }
    if (whole && c >= n - kHs) {
      line[c - n] = p[0];
      line[pl + c - n] = p[1];
    }
  } else if (c == 0 || c == n - 1) {
    const dw zero{0.f, 0.f};
    for (int h = 0; h < 4; ++h)
      if (c == (h < 2 ? 0 : n - 1)) {
        const int t = h < 2 ? h - 2 : n + h - 2;
        line[t] = pack(lo_of(p[0]), u_of(h));
        line[pl + t] = pack(zero, hi_of(p[1]));
      }
  }
}

template <int DIR>
__global__ void __launch_bounds__(kSplitWarps * 32, 1) k_line_split(const __grid_constant__ SplitLineParams P) {
  extern __shared__ __align__(16) unsigned char smem_line[];
  __shared__ RowS rows[kLineMax];  // x
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
  const int shift = whole ? kHs : 6 - p0;  // cell c of a line is at [c + shift]
  const size_t pl = (size_t)nl_cta * P.lp;
  dw2* buf[2] = {reinterpret_cast<dw2*>(smem_line), reinterpret_cast<dw2*>(smem_line) + 2 * pl};
  double* f64 = reinterpret_cast<double*>(smem_line + 4 * pl * sizeof(dw2));
  RowS* rz = reinterpret_cast<RowS*>(f64 + 4 * pl);  // z: of interface i at [i - first(0)]
  auto at = [&](int l) { return (size_t)l * P.lp + shift; };
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int l = w / P.runs, rn = w - l * P.runs;  // the warp's line and run
  const int c0 = first(0) + rn * P.run, c1 = min(c0 + P.run, past(0));
  const bool live = l < nl && c0 < c1;

  // row constants and wall ratios (backgrounds only: the kernel before it does not write them)
  if (DIR == MW_DIR_X) {
    load_pow_tables(pow_tables);
    __syncthreads();
    if (threadIdx.x < nl) {
      const int k = l0 + threadIdx.x + kHs;
      const double rt = MW_AT(a.hytc, k, P.nlines + 2 * kHs);
      rows[threadIdx.x] = row_consts(MW_AT(a.hyc, k, P.nlines + 2 * kHs), rt, kC0 * pow_gamma(rt, pow_tables));
    }
  } else {
    if (threadIdx.x < 4) {
      const int h = threadIdx.x < 2 ? threadIdx.x : n + threadIdx.x, src = threadIdx.x < 2 ? kHs : n + kHs - 1;
      hr[threadIdx.x] = MW_AT(a.hyc, h, n + 2 * kHs) / MW_AT(a.hyc, src, n + 2 * kHs);
    }
    for (int i = first(0) + threadIdx.x; i <= past(0); i += blockDim.x)
      rz[i - first(0)] = row_consts(MW_AT(a.hyi, i, n + 1), MW_AT(a.hyti, i, n + 1), MW_AT(a.hypi, i, n + 1));
    __syncthreads();  // hr
  }
  overlap_wait();
  if (gridDim.x <= kLineFewCtas) overlap_next();
  {
    const int ca = whole ? 0 : (DIR == MW_DIR_X ? p0 - 6 : max(p0 - 6, 0));
    const int cb = whole ? n : (DIR == MW_DIR_X ? p1 + 6 : min(p1 + 6, n));
    each_cell4<DIR>(P, l0, nl, ca, cb, [&](int ll, int c, long long o) {
      double v[4];
      dw2 p[2];
#pragma unroll
      for (int q = 0; q < 4; ++q) v[q] = MW_LG(a.in, q * P.plane + o);
      pack4(v, p);
#pragma unroll
      for (int q = 0; q < 4; ++q) f64[q * pl + at(ll) + c] = v[q];
      put_pairs<DIR>(buf[0] + at(ll), pl, c, n, whole, p, [&](int h) { return from_f64(v[UMOM] * hr[h]); });
    });
  }
  const int i = c0 + lane;  // the lane's interface and the cell to its right
  const Hv2 hv = make_hv2(ld(P.hv12));
  dw sw{0.f, 0.f};
  if (a.srcw && live && lane < 31 && i < c1) {
    const int c = DIR == MW_DIR_Z ? i : (i < 0 ? i + n : (i >= n ? i - n : i));
    const long long o = DIR == MW_DIR_X ? (long long)(l0 + l) * n + c : (long long)c * P.nlines + l0 + l;
    sw = mul(from_f64(MW_AT(a.srcw, o, (long long)n * P.nlines)), ld(P.d12));
  }
  __syncthreads();

  double iv[4];  // the direction's initial state at the lane's cell
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const bool pairs = s == 0 && !a.s1;  // the first stage's result is a pair unless it is asked for
    const bool out64 = s == 2 || (s == 0 ? a.s1 : a.s2);
    if (live) {
      const dw2* src = buf[s & 1] + at(l);
      dw2* dst = buf[(s + 1) & 1] + at(l);
      const int ii = min(max(i, first(s)), past(s));  // lanes beyond the stage's cells repeat its last interface
      dw2 t[2][4], F[2];
#pragma unroll
      for (int pr = 0; pr < 2; ++pr)
#pragma unroll
        for (int j = 0; j < 4; ++j) t[pr][j] = src[pr * pl + ii - 2 + j];
      if (DIR == MW_DIR_X)
        flux_x2(t, rows[l], hv, F);
      else
        flux_z2(t, rz[ii - first(0)], hv, ii == 0 || ii == n, F);
      dw2 G[2];  // the flux of the next interface
#pragma unroll
      for (int pr = 0; pr < 2; ++pr) {
        G[pr].h.x = __shfl_down_sync(0xffffffffu, F[pr].h.x, 1);
        G[pr].h.y = __shfl_down_sync(0xffffffffu, F[pr].h.y, 1);
        G[pr].l.x = __shfl_down_sync(0xffffffffu, F[pr].l.x, 1);
        G[pr].l.y = __shfl_down_sync(0xffffffffu, F[pr].l.y, 1);
      }
      if (lane < 31 && i >= max(c0, first(s)) && i < min(c1, past(s))) {
        if (s == 0) {
#pragma unroll
          for (int q = 0; q < 4; ++q) iv[q] = f64[q * pl + at(l) + i];
        }
        dw2 dF[2] = {sub2(F[0], G[0]), sub2(F[1], G[1])};
        dw dww = lo_of(dF[1]);
        if (DIR == MW_DIR_Z) dww = sub(dww, mul(lo_of(t[0][2]), ld(P.gz12)));
        if (a.srcw) dww = add(dww, sw);
        dF[1].h.x = dww.h;
        dF[1].l.x = dww.l;
        double v[4];
        dw2 r[2];
        if (pairs) {
          const dw2 ip[2] = {t[0][2], t[1][2]};
          update_pairs(ip, dF, ld(P.c12), r);
          put_pairs<DIR>(dst, pl, i, n, whole, r, [&](int h) { return mul(hi_of(r[0]), from_f64(hr[h])); });
        } else {
          update_f64(iv, dF, P.c12s[s], v);
          if (out64) {
#pragma unroll
            for (int q = 0; q < 4; ++q) f64[q * pl + at(l) + i] = v[q];
          }
          if (s < 2) {
            pack4(v, r);
            put_pairs<DIR>(dst, pl, i, n, whole, r, [&](int h) { return from_f64(v[UMOM] * hr[h]); });
          }
        }
        const bool edge = i >= p0 && i < p1 && (DIR == MW_DIR_X ? (i < kHs || i >= n - kHs) : (i == 0 || i == n - 1));
        if (edge) {
          const int line = DIR == MW_DIR_X ? l0 + l : l0 + l + kHs;
          if (s == 0 && a.halo_in) halo_out<DIR>(P, a.halo_in, line, i, iv, hr);
          if (s == 1 && a.halo_tmp) halo_out<DIR>(P, a.halo_tmp, line, i, v, hr);
        }
      }
    }
    __syncthreads();
    if (s == 2) overlap_next();  // at the latest (kLineFewCtas)
    double* g = s == 0 ? a.s1 : (s == 1 ? a.s2 : a.out);
    if (g) {
      each_cell4<DIR>(P, l0, nl, p0, p1, [&](int ll, int c, long long o) {
#pragma unroll
        for (int q = 0; q < 4; ++q) MW_LG(g, q * P.plane + o) = f64[q * pl + at(ll) + c];
      });
      if (s < 2) __syncthreads();  // the next stage's values go to the same place
    }
  }
  if (DIR == MW_DIR_Z && blockIdx.x == 0 && threadIdx.x < 8) halo_corners(P, hr);
}

template <int DIR>
int launch_split_line_t(const SplitLineParams& P, int ctas, int threads, size_t smem, bool overlap, cudaStream_t stream) {
  static std::atomic<int> done[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(MW_ERR_CUDA, "cudaGetDevice failed");
  if (dev < 0 || dev >= 64 || !done[dev].load(std::memory_order_relaxed)) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_line_split<DIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLineSmem);
    if (e != cudaSuccess) return fail(MW_ERR_CUDA, "line kernel shared memory: %s", cudaGetErrorString(e));
    if (dev >= 0 && dev < 64) done[dev].store(1, std::memory_order_relaxed);
  }
  return launch_overlapping(k_line_split<DIR>, dim3((unsigned)ctas), threads, smem, stream, overlap, "split line kernel",
                            P);
}

}  // namespace

int line_split_plan(int nx, int nz, LinePlan* plan) {
  *plan = LinePlan();
  if ((long long)nx * nz > kSplitLineCellsMax || std::max(nx, nz) > kSplitLineMax) return MW_OK;
  int sms = 0;
  const int st = line_sms(&sms);
  if (st) return st;
  *plan = line_plan(kSplitLines, nx, nz, sms);
  return MW_OK;
}

int launch_line_split(const LinePlan& plan, int nx, int nz, double dx, double dz, double dt_full, double dt,
                      const LineArgs& a, int direction, bool overlap, cudaStream_t stream) {
  SplitLineParams P;
  P.a = a;
  const bool isx = direction == MW_DIR_X;
  const double d = isx ? dx : dz;
  P.hv12 = split_host(12.0 * (-kHvBeta * d / (16 * dt_full)));
  P.d12 = split_host(12.0 * d);
  P.gz12 = split_host(12.0 * dz * kGrav);
  P.c12 = split_host(dt / 3 / (12.0 * d));
  for (int s = 0; s < 3; ++s) {
    const double c = dt / (3 - s) / (12.0 * d);
    P.c12s[s] = c * kTwoPow896;  // exact: a power-of-two scale
    MW_REQUIRE(std::isfinite(P.c12s[s]), MW_ERR_INVALID_ARG,
               "dt_stage / (12 d) = %g is above the split form's range (use the native FP64 mode)", c);
  }
  const LineSpread& sp = isx ? plan.x : plan.z;
  MW_REQUIRE(sp.pieces == 1 || a.in != a.out, MW_ERR_ALIAS, "a direction of cut lines needs another array for its result");
  int ctas, threads;
  set_line_geom(&P, sp, nx, nz, isx, &ctas, &threads);
  const size_t smem = line_smem(kSplitLines, P.lp, P.log_lines, isx);
  return isx ? launch_split_line_t<MW_DIR_X>(P, ctas, threads, smem, overlap, stream)
             : launch_split_line_t<MW_DIR_Z>(P, ctas, threads, smem, overlap, stream);
}

#if MW_CHECK
MW_OOB_COUNTER(oob_count_split_line)
#endif

}  // namespace mw
