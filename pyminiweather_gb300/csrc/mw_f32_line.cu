// mw_f32_line.cu -- the three RK stages of one direction in one launch, for
// grids whose lines fit a CTA (FP32 form).
//
// As mw_split_line.cu: whole lines or pieces of lines in shared memory, a warp
// per run of a line, a lane per interface and the cell to its right, the
// launches of a call overlapping; the arithmetic is that of the direction
// kernels (mw_f32_dir.cu), value for value.  Those fill and drain a pipeline per
// thread (z) or work through long runs (x), which takes a launch 8 us or more
// however small the grid; here a cell is one lane's work (100x50 15.6 -> 7.9 us a
// step, 512x256 19.1 -> 12.5), at the price of four shared-memory reads and both
// neighbours' second differences per cell, which larger grids pay for (700x500
// 25.1 -> 28.1).  A cell is a float4 in shared memory, twice (a stage's input and
// its result).
#include <algorithm>
#include <atomic>

#include "mw_common.cuh"
#include "mw_f32_dir.cuh"
#include "mw_f32_flux.cuh"
#include "mw_line.cuh"

namespace mw {
namespace f32 {
namespace {

constexpr int kF32Warps = 32;  // most per CTA, at up to 64 registers a thread
constexpr LineKind kF32Lines = {1, 1, {0, kF32Warps, 0}, {0, 64, 0}, 1, 32, sizeof(Row), 0.4};

struct LineF32Params : LineShape {
  F32DirArgs a;
  Consts k;
};

__device__ __forceinline__ float4 as_float4(const Vars& v) { return make_float4(v.a.x, v.a.y, v.b.x, v.b.y); }
__device__ __forceinline__ Vars as_vars(float4 v) { return {make_float2(v.x, v.y), make_float2(v.z, v.w)}; }

// Stores cell c of a line and the halo cells it is the source of, by the rules of put in mw_fp64_line.cu.
template <int DIR>
__device__ __forceinline__ void put(float4* line, int c, int n, bool whole, const Vars& v, const double* hr) {
  line[c] = as_float4(v);
  if (DIR == MW_DIR_X) {
    if (whole && c < kHs) line[n + c] = as_float4(v);
    if (whole && c >= n - kHs) line[c - n] = as_float4(v);
  } else {
    if (c == 0)
      for (int h = 0; h < 2; ++h) line[h - 2] = as_float4(wall_halo(v, hr, h));
    if (c == n - 1)
      for (int h = 2; h < 4; ++h) line[n + h - 2] = as_float4(wall_halo(v, hr, h));
  }
}

// The halo cells that cell c of a line is the source of, in a global array.
template <int DIR>
__device__ __forceinline__ void halo_out(const LineF32Params& P, float* g, int line, int c, const Vars& v,
                                         const double* hr) {
  const int n = P.n;
  if (DIR == MW_DIR_X) {
    const long long row = (long long)(line + kHs) * P.pitch;
    for (int q = 0; q < 4; ++q) {
      if (c < kHs) MW_LG(g, q * P.plane + row + n + kHs + c) = get(v, q);
      if (c >= n - kHs) MW_LG(g, q * P.plane + row + c - n + kHs) = get(v, q);
    }
  } else {
    for (int h = 0; h < 4; ++h)
      if (c == (h < 2 ? 0 : n - 1)) {
        const Vars w = wall_halo(v, hr, h);
        for (int q = 0; q < 4; ++q) MW_LG(g, q * P.plane + (long long)(h < 2 ? h : n + h) * P.pitch + line) = get(w, q);
      }
  }
}

template <int DIR>
__global__ void __launch_bounds__(kF32Warps * 32, 1) k_line_f32(const __grid_constant__ LineF32Params P) {
  extern __shared__ __align__(16) unsigned char smem_line[];
  __shared__ Row rows[kLineMax];  // x
  __shared__ double hr[4];
  const F32DirArgs& a = P.a;
  const int n = P.n, nl_cta = 1 << P.log_lines;
  const int group = blockIdx.x / P.pieces, pc = blockIdx.x - group * P.pieces;
  const int l0 = group << P.log_lines, nl = min(nl_cta, P.nlines - l0);
  const bool whole = P.pieces == 1;
  const int p0 = pc * P.piece, p1 = min(p0 + P.piece, n);  // the CTA's cells
  // first and last + 1 cell of a stage's result that the next stages need of this piece
  auto first = [&](int s) { return whole ? 0 : (DIR == MW_DIR_X ? p0 - 4 + 2 * s : max(p0 - 4 + 2 * s, 0)); };
  auto past = [&](int s) { return whole ? n : (DIR == MW_DIR_X ? p1 + 4 - 2 * s : min(p1 + 4 - 2 * s, n)); };
  const int shift = whole ? kHs : 6 - p0;  // cell c of a line is at [c + shift]
  const int pl = nl_cta * P.lp;
  float4* buf[2] = {reinterpret_cast<float4*>(smem_line) + shift, reinterpret_cast<float4*>(smem_line) + pl + shift};
  Row* rz = reinterpret_cast<Row*>(reinterpret_cast<float4*>(smem_line) + 2 * pl);  // z: of interface i at [i - first(0)]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int l = w / P.runs, rn = w - l * P.runs;  // the warp's line and run
  const int c0 = first(0) + rn * P.run, c1 = min(c0 + P.run, past(0));
  const bool live = l < nl && c0 < c1;

  // row constants and wall ratios (backgrounds only: the kernel before it does not write them)
  if (DIR == MW_DIR_X) {
    if (threadIdx.x < nl) {
      const int k = l0 + threadIdx.x + kHs;
      rows[threadIdx.x] = row_x(MW_AT(a.hyc, k, P.nlines + 2 * kHs), MW_AT(a.hytc, k, P.nlines + 2 * kHs));
    }
  } else {
    if (threadIdx.x < 4) {
      const int h = threadIdx.x < 2 ? threadIdx.x : n + threadIdx.x, src = threadIdx.x < 2 ? kHs : n + kHs - 1;
      hr[threadIdx.x] = MW_AT(a.hyc, h, n + 2 * kHs) / MW_AT(a.hyc, src, n + 2 * kHs);
    }
    for (int i = first(0) + threadIdx.x; i <= past(0); i += blockDim.x)
      rz[i - first(0)] = row_z(MW_AT(a.hyi, i, n + 1), MW_AT(a.hyti, i, n + 1), MW_AT(a.hypi, i, n + 1));
    __syncthreads();  // hr
  }
  overlap_wait();
  if (gridDim.x <= kLineFewCtas) overlap_next();
  {
    const int ca = whole ? 0 : (DIR == MW_DIR_X ? p0 - 6 : max(p0 - 6, 0));
    const int cb = whole ? n : (DIR == MW_DIR_X ? p1 + 6 : min(p1 + 6, n));
    each_cell4<DIR>(P, l0, nl, ca, cb, [&](int ll, int c, long long o) {
      const Vars v = {make_float2(MW_LG(a.in, o), MW_LG(a.in, P.plane + o)),
                      make_float2(MW_LG(a.in, 2 * P.plane + o), MW_LG(a.in, 3 * P.plane + o))};
      put<DIR>(buf[0] + ll * P.lp, c, n, whole, v, hr);
    });
  }
  const int i = c0 + lane;  // the lane's interface and the cell to its right
  float sw = 0.0f;
  if (a.srcw && live && lane < 31 && i < c1) {
    const int c = DIR == MW_DIR_Z ? i : (i < 0 ? i + n : (i >= n ? i - n : i));
    const long long o = DIR == MW_DIR_X ? (long long)(l0 + l) * n + c : (long long)c * P.nlines + l0 + l;
    sw = split::d2f(MW_AT(a.srcw, o, (long long)n * P.nlines));
  }
  __syncthreads();

  Vars iv;  // the direction's initial state at the lane's cell
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    if (live) {
      const float4* src = buf[s & 1] + l * P.lp;
      float4* dst = buf[(s + 1) & 1] + l * P.lp;
      const int ii = min(max(i, first(s)), past(s));  // lanes beyond the stage's cells repeat its last interface
      Vars t[4], e0, q0, e1, q1;
#pragma unroll
      for (int j = 0; j < 4; ++j) t[j] = as_vars(src[ii - 2 + j]);
      cell_eq(t[0], t[1], t[2], e0, q0);
      cell_eq(t[1], t[2], t[3], e1, q1);
      const Vars A = {f2add(q0.a, q1.a), f2add(q0.b, q1.b)}, D = {f2sub(e1.a, e0.a), f2sub(e1.b, e0.b)};
      bool far = false;
      const Row row = DIR == MW_DIR_X ? rows[l] : rz[ii - first(0)];
      Vars F = flux<DIR, false>(A, D, row, P.k, ii == 0 || ii == n, far);
      if (__any_sync(0xffffffffu, far)) F = flux<DIR, true>(A, D, row, P.k, ii == 0 || ii == n, far);
      const Vars G = {make_float2(__shfl_down_sync(0xffffffffu, F.a.x, 1), __shfl_down_sync(0xffffffffu, F.a.y, 1)),
                      make_float2(__shfl_down_sync(0xffffffffu, F.b.x, 1), __shfl_down_sync(0xffffffffu, F.b.y, 1))};
      if (lane < 31 && i >= max(c0, first(s)) && i < min(c1, past(s))) {
        if (s == 0) iv = t[2];
        Vars v;
        if (DIR == MW_DIR_X && !a.srcw) {
          v = update(iv, F, G, P.k.c[s]);
        } else {
          float g = P.k.dt[s] * sw;
          if (DIR == MW_DIR_Z) g = fmaf(P.k.gdt[s], t[2].a.x, g);
          v = update(iv, F, G, P.k.c[s], g);
        }
        put<DIR>(dst, i, n, whole, v, hr);
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
    float* g = s == 1 ? a.s2 : (s == 2 ? a.out : nullptr);
    if (g)
      each_cell4<DIR>(P, l0, nl, p0, p1, [&](int ll, int c, long long o) {
        const Vars v = as_vars(buf[(s + 1) & 1][ll * P.lp + c]);
#pragma unroll
        for (int q = 0; q < 4; ++q) MW_LG(g, q * P.plane + o) = get(v, q);
      });
  }
  // the four x-halo columns of the wall halo rows, from the halo columns' own first and last rows
  if (DIR == MW_DIR_Z && blockIdx.x == 0 && threadIdx.x < 8) {
    float* g = threadIdx.x < 4 ? a.halo_in : a.halo_tmp;
    const int col = (threadIdx.x & 2) ? P.nlines + (threadIdx.x & 3) : (threadIdx.x & 1);
    if (g)
      for (int top = 0; top < 2; ++top) {
        auto at = [&](int q) { return MW_LG(g, q * P.plane + (long long)(top ? n + kHs - 1 : kHs) * P.pitch + col); };
        const Vars v = {make_float2(at(0), at(1)), make_float2(at(2), at(3))};
        for (int h = 2 * top; h < 2 * top + 2; ++h) {
          const Vars hv = wall_halo(v, hr, h);
          for (int q = 0; q < 4; ++q) MW_LG(g, q * P.plane + (long long)(h < 2 ? h : n + h) * P.pitch + col) = get(hv, q);
        }
      }
  }
}

template <int DIR>
int launch_t(const LineF32Params& P, int ctas, int threads, size_t smem, bool overlap, cudaStream_t stream) {
  static std::atomic<int> done[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return fail(MW_ERR_CUDA, "cudaGetDevice failed");
  if (dev < 0 || dev >= 64 || !done[dev].load(std::memory_order_relaxed)) {
    const cudaError_t e =
        cudaFuncSetAttribute(k_line_f32<DIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLineSmem);
    if (e != cudaSuccess) return fail(MW_ERR_CUDA, "line kernel shared memory: %s", cudaGetErrorString(e));
    if (dev >= 0 && dev < 64) done[dev].store(1, std::memory_order_relaxed);
  }
  return launch_overlapping(k_line_f32<DIR>, dim3((unsigned)ctas), threads, smem, stream, overlap, "FP32 line kernel", P);
}

}  // namespace
}  // namespace f32

int line_f32_plan(int nx, int nz, LinePlan* plan) {
  *plan = LinePlan();
  if ((long long)nx * nz > kF32LineCellsMax) return MW_OK;
  int sms = 0;
  const int st = line_sms(&sms);
  if (st) return st;
  *plan = line_plan(f32::kF32Lines, nx, nz, sms);
  return MW_OK;
}

int launch_line_f32(const LinePlan& plan, int nx, int nz, double dx, double dz, double dt_full, double dt,
                    const F32DirArgs& d, int direction, bool overlap, cudaStream_t stream) {
  using namespace f32;
  const bool isx = direction == MW_DIR_X;
  LineF32Params P;
  P.a = d;
  P.k = step_consts(isx ? dx : dz, dt_full, dt);
  const LineSpread& sp = isx ? plan.x : plan.z;
  MW_REQUIRE(sp.pieces == 1 || d.in != d.out, MW_ERR_ALIAS, "a direction of cut lines needs another array for its result");
  int ctas, threads;
  set_line_geom(&P, sp, nx, nz, isx, &ctas, &threads);
  const size_t smem = line_smem(kF32Lines, P.lp, P.log_lines, isx);
  return isx ? launch_t<MW_DIR_X>(P, ctas, threads, smem, overlap, stream)
             : launch_t<MW_DIR_Z>(P, ctas, threads, smem, overlap, stream);
}

#if MW_CHECK
MW_OOB_COUNTER(oob_count_f32_line)
#endif

}  // namespace mw
