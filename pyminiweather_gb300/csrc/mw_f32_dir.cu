// mw_f32_dir.cu -- FP32 form: the three RK stages of one direction in one
// launch (two launches per step: evolve, pyminiweather/solve/step.py:85-143),
// single grids and ensembles.
//
// The scheme is split by direction, so the stages of a direction couple only
// the cells of a row (x) or a column (z): out(k) needs the initial state at
// k - 6 .. k + 6.  One launch per stage is bound by HBM (256 B per cell-step:
// each stage reads and writes the state); here a direction reads the state
// once and writes it once, 64 B per cell-step and 16 B more where state_tmp is
// asked for, and what bounds it is FP32 issue and HBM about equally.
//
// z: a thread marches down a column.  Each stage is a stream: row k + 1 of its
// input yields e, q of row k, the flux at interface k and row k - 1 of its
// output, which is the next stage's input.  The initial state comes through a
// ring of 16 rows per thread in shared memory, filled nine rows ahead by
// asynchronous copies that each thread issues and awaits itself (no CTA
// barrier, any alignment), which also holds the rows back to the third stage's
// initial values, six behind.
// x: a warp takes a run of a row, V consecutive cells per lane, through the
// three stages in registers; what a lane needs of its neighbours' cells comes
// by shuffles.  The run's cells and six to each side are staged through shared
// memory by asynchronous copies, one run ahead.
// Arithmetic: the two stencils by second differences (e = s(k-1) - 2 s(k) +
// s(k+1), q = s - e / 6: twice the interpolation is q(k-1) + q(k), the third
// difference e(k) - e(k-1)), the variables in pairs (DENS, UMOM) and (WMOM,
// RHOT) through packed FP32 instructions (mw_f32_flux.cuh).
#include <algorithm>
#include <atomic>
#include <mutex>

#include "mw_common.cuh"
#include "mw_ensemble.cuh"
#include "mw_f32_dir.cuh"
#include "mw_f32_flux.cuh"

namespace mw {
namespace f32 {

constexpr int kZCols = 128;    // columns per z CTA (single grid)
constexpr int kRing = 16;      // rows of a thread's ring
constexpr int kAhead = 9;      // rows loaded ahead
constexpr int kLag = 6;        // row r of the state comes in when row r - 6 of the result goes out
constexpr int kZTileMax = 512; // rows per z CTA
constexpr int kXWarps = 4;     // warps per x CTA
// A launch lets the next one in only when it ends: earlier, its CTAs would share
// SMs with the next one's, which stay there (2501x1251: 98 us a step with every
// launch doing so at its head, 79 with none; 20001x1, of under a CTA per SM, 16.2
// either way).

struct Args {
  int nx, nz, pitch;
  long long plane;
  const double* hyc;
  const double* hytc;
  const double* hyi;
  const double* hyti;
  const double* hypi;
  const double* srcw;
  const float* in;
  float* out;
  float* s2;
  float* halo_in;
  float* halo_tmp;
  Consts k;
};
#define MW_G(p, off) MW_AT((p), (off), 4 * a.plane)

__device__ __forceinline__ void copy4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// ---- z ---------------------------------------------------------------------
// One stage's stream: the two latest rows it has, e and q of the latest but
// one, and the flux at the interface below that row.
struct Stream {
  Vars s0, s1, e, q, F;
};

// What row `idx` of a stage's input yields: the row as it enters the stream,
// its e, q and flux, and row idx - 2 of the stage's result (src: dt_stage times
// the forcing of its w).  WALL: the row may
// be a wall's (the rows that follow nz - 1 are built from the stream); without
// it 2 <= idx < nz holds.
struct Pushed {
  Vars v, e, q, F, o;
};
template <bool WALL, bool ANY>
__device__ __forceinline__ Pushed push(const Stream& st, Vars v, int idx, int nz, const double* hr, const Row& row,
                                       const Consts& k, int stage, const Vars& init, float src, bool& far) {
  if (WALL) {
    if (idx == nz) v = wall_halo(st.s1, hr, 2);
    if (idx == nz + 1) v = wall_halo(st.s0, hr, 3);
  }
  Pushed r;
  r.v = v;
  cell_eq(st.s0, st.s1, v, r.e, r.q);
  const Vars A = {f2add(st.q.a, r.q.a), f2add(st.q.b, r.q.b)}, D = {f2sub(r.e.a, st.e.a), f2sub(r.e.b, st.e.b)};
  r.F = flux<MW_DIR_Z, ANY>(A, D, row, k, WALL && (idx == 1 || idx == nz + 1), far);
  // gravity on the forcing's rho' (interpolate.py:248-250) and the source
  r.o = update(init, st.F, r.F, k.c[stage], fmaf(k.gdt[stage], st.s0.a.x, src));
  return r;
}
template <bool WALL>
__device__ __forceinline__ void commit(Stream& st, const Pushed& r, int idx, const double* hr) {
  st = {st.s1, r.v, r.e, r.q, r.F};
  if (WALL && idx == 0) {  // the rows below the wall
    st.s0 = wall_halo(r.v, hr, 1);
    cell_eq(wall_halo(r.v, hr, 0), st.s0, r.v, st.e, st.q);
  }
}

template <int NC>
struct SmemZ {
  float ring[kRing][4][NC];
  double hr[4];
};

// Rows [z0, z1) of the columns [cb NC, cb NC + NC); every thread of the CTA
// calls it (one barrier after the row table is formed).  tab: z1 - z0 + 17 rows
// of shared memory.  SRC: the forcing of w comes through a ring of its own (srcs,
// kRing rows of NC) beside the state's: read where the three stages add it, it
// stood in each one's way (2501x1251: 175 us a step, 127 here, 82 without forcing).
// TMP: the second stage is stored too.  Without it the march is unrolled by four
// (8192x2048: 145 against 169 us, the streams' rows keep their registers); with
// it the extra stores bound the pass and the compact loop does better (190
// against 198 us).
template <int NC, bool SRC, bool TMP>
__device__ __forceinline__ void z_march(const Args& a, int cb, int z0, int z1, SmemZ<NC>& sm, Row* tab,
                                        double* srcs = nullptr) {
  const int a0 = max(z0 - 6, 0), last = z1 - 1 + kLag;  // first row in; last iteration
  const int t = threadIdx.x, nz = a.nz;
  for (int i = t; i <= last - a0 + 5; i += NC) {  // interface a0 - 6 + i, clamped where nothing uses it
    const int k = min(max(a0 - 6 + i, 0), nz);
    tab[i] = row_z(MW_AT(a.hyi, k, nz + 1), MW_AT(a.hyti, k, nz + 1), MW_AT(a.hypi, k, nz + 1));
  }
  if (t < 4) {
    const int h = t < 2 ? t : nz + t, src = t < 2 ? kHs : nz + kHs - 1;
    sm.hr[t] = MW_AT(a.hyc, h, nz + 2 * kHs) / MW_AT(a.hyc, src, nz + 2 * kHs);
  }
  __syncthreads();
  overlap_wait();
  const int c = cb * NC + t;
  // the wall halo rows (arrays that ask for them): of the initial state here, and of the x-halo columns of
  // both arrays from the halo columns' own first and last rows
  auto put_halo = [&](float* g, int col, bool top, const Vars& v) {
    for (int h = 0; h < 2; ++h) {
      const Vars w = wall_halo(v, sm.hr, (top ? 2 : 0) + h);
      for (int q = 0; q < 4; ++q)
        MW_G(g, q * a.plane + (long long)((top ? nz + kHs : 0) + h) * a.pitch + col) = get(w, q);
    }
  };
  auto column = [&](const float* g, int col, int row) {
    auto at = [&](int q) { return MW_G(g, q * a.plane + (long long)(row + kHs) * a.pitch + col); };
    return Vars{make_float2(at(0), at(1)), make_float2(at(2), at(3))};
  };
  for (int top = 0; top < 2; ++top) {
    if (top ? z1 != nz : z0 != 0) continue;
    const int row = top ? nz - 1 : 0;
    if (a.halo_in && c < a.nx) put_halo(a.halo_in, c + kHs, top, column(a.in, c + kHs, row));
    if (cb == 0 && t < 4) {
      const int col = t < 2 ? t : a.nx + t;
      if (a.halo_in) put_halo(a.halo_in, col, top, column(a.halo_in, col, row));
      if (a.halo_tmp) put_halo(a.halo_tmp, col, top, column(a.halo_tmp, col, row));
    }
  }
  const bool act = c < a.nx;  // the others march the last column and store nothing
  const int cc = min(c, a.nx - 1);
  // element (row a0 + r, this column) of variable q of a state array: a base that is uniform in the CTA and a 32-bit
  // byte offset (the host keeps a tile's rows below 2^32 bytes)
  const long long base = (long long)(a0 + kHs) * a.pitch + kHs;
  const unsigned pitch4 = 4u * (unsigned)a.pitch;
  auto elem = [&](auto* g, int q, unsigned off) {
#if MW_CHECK
    return &MW_G(g, q * a.plane + base + off / 4);
#else
    return g + (q * a.plane + base) + off / 4;
#endif
  };
  unsigned off_in = 4u * (unsigned)cc;  // of the next row to load
  auto load = [&](int r) {  // row r into its slot (each row is one group of copies)
    if (r < nz && r <= z1 + 5) {
#pragma unroll
      for (int q = 0; q < 4; ++q) copy4(&sm.ring[r & (kRing - 1)][q][t], elem(a.in, q, off_in));
      if (SRC) copy8(&srcs[(r & (kRing - 1)) * NC + t], &MW_AT(a.srcw, (long long)r * a.nx + cc, (long long)a.nx * nz));
    }
    off_in += pitch4;
    copies_commit();
  };
  auto ring = [&](int r) {
    const float(*w)[NC] = sm.ring[r & (kRing - 1)];
    return Vars{make_float2(w[0][t], w[1][t]), make_float2(w[2][t], w[3][t])};
  };
  auto store = [&](float* g, unsigned off, const Vars& v) {
    *elem(g, 0, off) = v.a.x;
    *elem(g, 1, off) = v.a.y;
    *elem(g, 2, off) = v.b.x;
    *elem(g, 3, off) = v.b.y;
  };
  for (int r = a0; r < a0 + kAhead; ++r) load(r);
  const Vars zero = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
  Stream st[3];
#pragma unroll
  for (int s = 0; s < 3; ++s) st[s] = {zero, zero, zero, zero, zero};
  auto iterate = [&](int r, auto wall) {
    constexpr bool W = decltype(wall)::value;
    load(r + kAhead);
    copies_wait<kAhead>();
    const Row* rw = tab + (r - a0);
    // row idx into stage s; its result's row idx - 2
    auto stage = [&](int s, const Vars& v, int idx, const Vars& init) {
      bool far = false;
      float src = 0.0f;
      if (SRC) {
        const int k = idx - 2;
        if (k >= a0 && k < nz) src = a.k.dt[s] * split::d2f(srcs[(k & (kRing - 1)) * NC + t]);
      }
      Pushed p = push<W, W>(st[s], v, idx, nz, sm.hr, rw[5 - 2 * s], a.k, s, init, src, far);
      if (!W && __any_sync(0xffffffffu, far))
        p = push<W, true>(st[s], v, idx, nz, sm.hr, rw[5 - 2 * s], a.k, s, init, src, far);
      commit<W>(st[s], p, idx, sm.hr);
      return p.o;
    };
    const Vars v1 = stage(0, ring(r), r, st[0].s0);
    const Vars v2 = stage(1, v1, r - 2, ring(r - 4));
    const Vars o = stage(2, v2, r - 4, ring(r - 6));
    const unsigned off = off_in - 16u * pitch4;  // row r - 6 (off_in is at row r + 10)
    if (TMP && act && r - 4 >= z0 && r - 4 < z1) store(a.s2, off + 2u * pitch4, v2);
    if (W && act && a.halo_tmp) {
      if (r - 4 == 0 && z0 == 0) put_halo(a.halo_tmp, c + kHs, false, v2);
      if (r - 4 == nz - 1 && z1 == nz) put_halo(a.halo_tmp, c + kHs, true, v2);
    }
    if (act && r - 6 >= z0) store(a.out, off, o);
  };
  int r = a0;
  const int fast0 = min(6, last + 1);
  for (; r < fast0; ++r) iterate(r, std::true_type{});
  const int fast1 = min(nz, last + 1);
  if (TMP) {
#pragma unroll 1
    for (; r < fast1; ++r) iterate(r, std::false_type{});
  } else {
#pragma unroll 4
    for (; r < fast1; ++r) iterate(r, std::false_type{});
  }
  for (; r <= last; ++r) iterate(r, std::true_type{});
  copies_wait<0>();
}

template <bool SRC, bool TMP>
__global__ void __launch_bounds__(kZCols, 4) k_dir_z_f32(const __grid_constant__ Args a, int tile, int tile0) {
  extern __shared__ __align__(16) unsigned char smem_f32[];
  SmemZ<kZCols>& sm = *reinterpret_cast<SmemZ<kZCols>*>(smem_f32);
  const int z0 = (tile0 + blockIdx.y) * tile;
  Row* tab = reinterpret_cast<Row*>(&sm + 1);
  z_march<kZCols, SRC, TMP>(a, blockIdx.x, z0, min(z0 + tile, a.nz), sm, tab, reinterpret_cast<double*>(tab + tile + 17));
}

// ---- x ---------------------------------------------------------------------
template <int V, bool SRC = false>
struct XBuf {
  float v[4][32 * V + 4];               // cells c0 - 6 + j of a run
  double src[SRC ? 32 * V + 2 : 1];     // their forcing of w
};
template <int V>
struct XBuf<V, false> {
  float v[4][32 * V + 4];
};
static_assert(sizeof(XBuf<4, true>) % 16 == 0 && sizeof(XBuf<8, true>) % 16 == 0, "buffers are read in float4");
constexpr int x_run_max(int V) { return 32 * V - 12; }

__device__ __forceinline__ Vars shfl_up(const Vars& v) {
  constexpr unsigned m = 0xffffffffu;
  return {make_float2(__shfl_up_sync(m, v.a.x, 1), __shfl_up_sync(m, v.a.y, 1)),
          make_float2(__shfl_up_sync(m, v.b.x, 1), __shfl_up_sync(m, v.b.y, 1))};
}
__device__ __forceinline__ Vars shfl_down(const Vars& v) {
  constexpr unsigned m = 0xffffffffu;
  return {make_float2(__shfl_down_sync(m, v.a.x, 1), __shfl_down_sync(m, v.a.y, 1)),
          make_float2(__shfl_down_sync(m, v.b.x, 1), __shfl_down_sync(m, v.b.y, 1))};
}

// Copies of the cells c0 - 6 .. c0 + len + 5 of row k (periodic) into b, one group.
template <int V, bool SRC = false>
__device__ __forceinline__ void x_load(const Args& a, int k, int c0, int len, XBuf<V, SRC>& b) {
  const int lane = threadIdx.x & 31;
  const long long row = (long long)(k + kHs) * a.pitch + kHs;
  if (c0 >= 6 && c0 + len + 6 <= a.nx) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int j = lane + 32 * i;
      if (j < len + 12)
#pragma unroll
        for (int q = 0; q < 4; ++q) copy4(&b.v[q][j], &MW_G(a.in, q * a.plane + row + (c0 - 6) + j));
      if constexpr (SRC)
        if (j < len + 12) copy8(&b.src[j], &MW_AT(a.srcw, (long long)k * a.nx + (c0 - 6) + j, (long long)a.nx * a.nz));
    }
  } else {
    for (int j = lane; j < len + 12; j += 32) {
      int c = c0 - 6 + j;
      if (a.nx < 12) {
        c %= a.nx;
        if (c < 0) c += a.nx;
      } else {
        c = c < 0 ? c + a.nx : (c >= a.nx ? c - a.nx : c);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) copy4(&b.v[q][j], &MW_G(a.in, q * a.plane + row + c));
      if constexpr (SRC) copy8(&b.src[j], &MW_AT(a.srcw, (long long)k * a.nx + c, (long long)a.nx * a.nz));
    }
  }
  copies_commit();
}

// One stage of a run: v from S and v, shuffles across the warp.  SRC: dt times src is added to rho w.
template <int V, bool ANY, bool SRC>
__device__ __forceinline__ void x_stage(Vars (&v)[V], const Vars (&S)[V], const Row& row, const Consts& k, float c,
                                        float dt, const float (&src)[V]) {
  auto upd = [&](int j, const Vars& Fp, const Vars& F) {
    return SRC ? update(S[j], Fp, F, c, dt * src[j]) : update(S[j], Fp, F, c);
  };
  const Vars m2 = shfl_up(v[V - 2]), m1 = shfl_up(v[V - 1]), p = shfl_down(v[0]);
  Vars e0, q0, Fp, F0;
  cell_eq(m2, m1, v[0], e0, q0);
  Vars before = m1;
  bool far = false;
#pragma unroll
  for (int j = 0; j < V; ++j) {
    const Vars cur = v[j];
    Vars e, q;
    cell_eq(before, cur, j + 1 < V ? v[j + 1] : p, e, q);
    const Vars A = {f2add(q0.a, q.a), f2add(q0.b, q.b)}, D = {f2sub(e.a, e0.a), f2sub(e.b, e0.b)};
    const Vars F = flux<MW_DIR_X, ANY>(A, D, row, k, false, far);
    if (j == 0)
      F0 = F;
    else
      v[j - 1] = upd(j - 1, Fp, F);
    Fp = F;
    e0 = e;
    q0 = q;
    before = cur;
  }
  v[V - 1] = upd(V - 1, Fp, shfl_down(F0));
}

// The run of `len` cells from c0 of row k, staged in b (which it reuses for its
// results); every lane of the warp calls it.
template <int V, bool SRC>
__device__ __forceinline__ void x_run(const Args& a, int k, int c0, int len, const Row& row,
                                      XBuf<V, SRC>& b) {
  const int lane = threadIdx.x & 31;
  const long long go = (long long)(k + kHs) * a.pitch + kHs + c0;
  Vars S[V], v[V];
#pragma unroll
  for (int g = 0; g < V; g += 4) {
    float4 w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) w[q] = *reinterpret_cast<const float4*>(&b.v[q][V * lane + g]);
    S[g] = {make_float2(w[0].x, w[1].x), make_float2(w[2].x, w[3].x)};
    S[g + 1] = {make_float2(w[0].y, w[1].y), make_float2(w[2].y, w[3].y)};
    S[g + 2] = {make_float2(w[0].z, w[1].z), make_float2(w[2].z, w[3].z)};
    S[g + 3] = {make_float2(w[0].w, w[1].w), make_float2(w[2].w, w[3].w)};
  }
#pragma unroll
  for (int j = 0; j < V; ++j) v[j] = S[j];
  float src[V];
  if constexpr (SRC) {  // the cells beyond the run and its neighbours' are not used
#pragma unroll
    for (int j = 0; j < V; ++j) src[j] = split::d2f(b.src[V * lane + j]);
  }
  auto stage_out = [&](float* g, bool halo) {  // cells c0 .. c0 + len - 1 of v through b to g
    __syncwarp();
#pragma unroll
    for (int h = 0; h < V; h += 4)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<float4*>(&b.v[q][V * lane + h]) =
            make_float4(get(v[h], q), get(v[h + 1], q), get(v[h + 2], q), get(v[h + 3], q));
    __syncwarp();
    if (g) {
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int j = lane + 32 * i;
        if (j < len)
#pragma unroll
          for (int q = 0; q < 4; ++q) MW_G(g, q * a.plane + go + j) = b.v[q][6 + j];
      }
    }
    if (halo && (c0 < kHs || c0 + len > a.nx - kHs))  // the periodic halo cells these cells are the source of
      for (int j = lane; j < len; j += 32) {
        const int c = c0 + j;
        for (int q = 0; q < 4; ++q) {
          if (c < kHs) MW_G(a.halo_tmp, q * a.plane + go - c0 + a.nx + c) = b.v[q][6 + j];
          if (c >= a.nx - kHs) MW_G(a.halo_tmp, q * a.plane + go - c0 + c - a.nx) = b.v[q][6 + j];
        }
      }
  };
  // |d| <= (4/3) max |(rho theta)'| / (rho theta)_bg at every interface: one check per stage decides for the run
  // (a NaN takes either path to a NaN)
  const float near = 0.0937f * 0.5f * row.RT;
#pragma unroll 1
  for (int s = 0; s < 3; ++s) {
    float m = 0.0f;
#pragma unroll
    for (int j = 0; j < V; ++j) m = fmaxf(m, fabsf(v[j].b.y));
    if (__any_sync(0xffffffffu, m > near))
      x_stage<V, true, SRC>(v, S, row, a.k, a.k.c[s], a.k.dt[s], src);
    else
      x_stage<V, false, SRC>(v, S, row, a.k, a.k.c[s], a.k.dt[s], src);
    if (s == 1 && (a.s2 || a.halo_tmp)) stage_out(a.s2, a.halo_tmp != nullptr);
  }
  stage_out(a.out, false);
}

// This row's periodic halo of the initial state (ics/bcs.py:35-39).
__device__ __forceinline__ void x_halo_in(const Args& a, int k) {
  const int lane = threadIdx.x & 31;
  if (a.halo_in && lane < 4) {  // columns 0, 1 <- nx, nx+1; nx+2, nx+3 <- 2, 3
    const long long row = (long long)(k + kHs) * a.pitch;
    const int dst = lane < 2 ? lane : a.nx + lane, src = lane < 2 ? a.nx + lane : lane;
#pragma unroll
    for (int q = 0; q < 4; ++q) MW_G(a.halo_in, q * a.plane + row + dst) = MW_G(a.in, q * a.plane + row + src);
  }
}

// Single grid: every warp takes a contiguous range of the row-major list of
// runs of `len` cells (nrun per row), the next run's copies in flight while it
// works on one.
template <int V, bool SRC>
__global__ void __launch_bounds__(32 * kXWarps, 4) k_dir_x_f32(const __grid_constant__ Args a, int nrun, int len,
                                                              long long total) {
  extern __shared__ __align__(16) unsigned char smem_f32[];
  XBuf<V, SRC>* buf = reinterpret_cast<XBuf<V, SRC>*>(smem_f32) + 2 * (threadIdx.x >> 5);
  const long long w = (long long)blockIdx.x * kXWarps + (threadIdx.x >> 5), nw = (long long)gridDim.x * kXWarps;
  const long long g0 = total * w / nw, g1 = total * (w + 1) / nw;
  int k = (int)(g0 / nrun), rn = (int)(g0 - (long long)k * nrun);
  Row row = {0.f, 0.f, 0.f, 0.f};
  if (g0 < g1) row = row_x(MW_AT(a.hyc, k + kHs, a.nz + 2 * kHs), MW_AT(a.hytc, k + kHs, a.nz + 2 * kHs));
  overlap_wait();
  if (g0 >= g1) return;
  x_load<V, SRC>(a, k, rn * len, min(len, a.nx - rn * len), buf[0]);
  int cur = 0;
  for (long long g = g0; g < g1; ++g) {
    const int kc = k, c0 = rn * len;
    if (++rn == nrun) {
      rn = 0;
      ++k;
    }
    __syncwarp();  // the other buffer's results are read
    if (g + 1 < g1) {
      x_load<V, SRC>(a, k, rn * len, min(len, a.nx - rn * len), buf[cur ^ 1]);
      copies_wait<1>();
    } else {
      copies_wait<0>();
    }
    __syncwarp();
    if (c0 == 0) x_halo_in(a, kc);
    x_run<V, SRC>(a, kc, c0, min(len, a.nx - c0), row, buf[cur]);
    if (k != kc && g + 1 < g1)
      row = row_x(MW_AT(a.hyc, k + kHs, a.nz + 2 * kHs), MW_AT(a.hytc, k + kHs, a.nz + 2 * kHs));
    cur ^= 1;
  }
}

// ---- ensembles -------------------------------------------------------------
__device__ __forceinline__ Args member_args(const EnsStageT<float>& es, int e) {
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
  a.in = es.init + m.state_off;
  a.out = es.out + m.state_off;
  a.s2 = es.s2 ? es.s2 + m.state_off : nullptr;
  a.halo_in = es.halo_in ? es.halo_in + m.state_off : nullptr;
  a.halo_tmp = es.halo_tmp ? es.halo_tmp + m.state_off : nullptr;
  const EnsMemberConsts* c = reinterpret_cast<const EnsMemberConsts*>(es.mconsts) + mconsts_index(es, e);
#pragma unroll
  for (int s = 0; s < 3; ++s) {  // the stages' entries follow one another
    a.k.c[s] = MW_AT(c, s, 3).c_f;
    a.k.dt[s] = MW_AT(c, s, 3).dt_f;
    a.k.gdt[s] = a.k.dt[s] * -float(kGrav);
  }
  a.k.HV = MW_AT(c, 0, 3).hv_f;
  return a;
}

// x items are rows (member, row), one per warp.
constexpr int kEnsV = 8;
__global__ void __launch_bounds__(32 * kXWarps, 4) k_ens_x_f32(EnsStageT<float> es) {
  extern __shared__ __align__(16) unsigned char smem_f32[];
  XBuf<kEnsV>* buf = reinterpret_cast<XBuf<kEnsV>*>(smem_f32) + 2 * (threadIdx.x >> 5);
  for (unsigned it = ens_take_warp(es.cursor); it < (unsigned)es.n_items; it = ens_take_warp(es.cursor)) {
    const int2 item = MW_AT(es.items, it, es.n_items);  // (member, row)
    const Args a = member_args(es, item.x);
    const int k = item.y, nrun = (a.nx + x_run_max(kEnsV) - 1) / x_run_max(kEnsV), len = (a.nx + nrun - 1) / nrun;
    __syncwarp();
    x_load<kEnsV>(a, k, 0, min(len, a.nx), buf[0]);
    const Row row = row_x(MW_AT(a.hyc, k + kHs, a.nz + 2 * kHs), MW_AT(a.hytc, k + kHs, a.nz + 2 * kHs));
    x_halo_in(a, k);
    int cur = 0;
    for (int c0 = 0; c0 < a.nx; c0 += len) {
      __syncwarp();
      if (c0 + len < a.nx) {
        x_load<kEnsV>(a, k, c0 + len, min(len, a.nx - c0 - len), buf[cur ^ 1]);
        copies_wait<1>();
      } else {
        copies_wait<0>();
      }
      __syncwarp();
      x_run<kEnsV, false>(a, k, c0, min(len, a.nx - c0), row, buf[cur]);
      cur ^= 1;
    }
  }
  ens_finish(es.cursor);
}

template <bool TMP>
__global__ void __launch_bounds__(kEnsZCols, 8) k_ens_z_f32(EnsStageT<float> es) {
  extern __shared__ __align__(16) unsigned char smem_f32[];
  SmemZ<kEnsZCols>& sm = *reinterpret_cast<SmemZ<kEnsZCols>*>(smem_f32);
  __shared__ unsigned slot[2];
  int parity = 0;
  for (unsigned it = ens_take_cta(es.cursor, slot, parity); it < (unsigned)(es.n_items * es.z_parts);
       it = ens_take_cta(es.cursor, slot, parity)) {
    const int2 item = MW_AT(es.items, it / es.z_parts, es.n_items);  // (member, column block + ncb * tile)
    const Args a = member_args(es, item.x);
    const int ncb = (a.nx + kEnsZCols - 1) / kEnsZCols;
    const int cb = item.y % ncb;
    int z0, z1;
    ens_part_rows(es, item.y / ncb, it % es.z_parts, a.nz, z0, z1);
    if (z0 >= z1) continue;
    z_march<kEnsZCols, false, TMP>(a, cb, z0, z1, sm, reinterpret_cast<Row*>(&sm + 1));
  }
  ens_finish(es.cursor);
}

size_t z_smem(int nc, int tile, bool src = false) {
  return (nc == kZCols ? sizeof(SmemZ<kZCols>) : sizeof(SmemZ<kEnsZCols>)) + sizeof(Row) * (tile + 17) +
         (src ? sizeof(double) * kRing * nc : 0);
}

// The kernels' shared-memory limits, raised once per device; the device's SMs
// and resident CTAs per SM of the two passes.
struct Device {
  std::mutex mu;
  std::atomic<int> sms{0};
  int x_ctas[2] = {0, 0}, z_ctas = 0;  // x: V = 4, 8
};
Device g_dev[64];

template <typename K>
cudaError_t raise_smem(K kernel, size_t bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

int device(Device** out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return fail(MW_ERR_CUDA, "no usable device");
  Device& d = g_dev[dev];
  *out = &d;
  if (d.sms.load(std::memory_order_acquire) > 0) return MW_OK;
  std::lock_guard<std::mutex> lock(d.mu);
  if (d.sms.load(std::memory_order_relaxed) > 0) return MW_OK;
  const size_t zs = z_smem(kZCols, kZTileMax), xs8 = sizeof(XBuf<8>) * 2 * kXWarps, xs4 = sizeof(XBuf<4>) * 2 * kXWarps;
  int sms = 0, x4 = 0, x8 = 0, z = 0;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = raise_smem(k_dir_z_f32<false, false>, zs);
  if (e == cudaSuccess) e = raise_smem(k_dir_z_f32<false, true>, zs);
  const size_t zs_src = z_smem(kZCols, kZTileMax, true);
  if (e == cudaSuccess) e = raise_smem(k_dir_z_f32<true, false>, zs_src);
  if (e == cudaSuccess) e = raise_smem(k_dir_z_f32<true, true>, zs_src);
  if (e == cudaSuccess) e = raise_smem(k_dir_x_f32<4, false>, xs4);
  if (e == cudaSuccess) e = raise_smem(k_dir_x_f32<4, true>, sizeof(XBuf<4, true>) * 2 * kXWarps);
  if (e == cudaSuccess) e = raise_smem(k_dir_x_f32<8, false>, xs8);
  if (e == cudaSuccess) e = raise_smem(k_dir_x_f32<8, true>, sizeof(XBuf<8, true>) * 2 * kXWarps);
  if (e == cudaSuccess) e = raise_smem(k_ens_x_f32, xs8);
  if (e == cudaSuccess) e = raise_smem(k_ens_z_f32<false>, z_smem(kEnsZCols, kEnsZTileMax));
  if (e == cudaSuccess) e = raise_smem(k_ens_z_f32<true>, z_smem(kEnsZCols, kEnsZTileMax));
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&x4, k_dir_x_f32<4, false>, 32 * kXWarps, xs4);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&x8, k_dir_x_f32<8, false>, 32 * kXWarps, xs8);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&z, k_dir_z_f32<false, false>, kZCols, zs);
  if (e != cudaSuccess) return fail(MW_ERR_CUDA, "FP32 kernel setup: %s", cudaGetErrorString(e));
  d.x_ctas[0] = std::max(1, x4);
  d.x_ctas[1] = std::max(1, x8);
  d.z_ctas = std::max(1, z);
  d.sms.store(sms, std::memory_order_release);
  return MW_OK;
}

}  // namespace f32

int launch_dir_f32(int nx, int nz, double dx, double dz, double dt_full, double dt, const F32DirArgs& d, int direction,
                   bool overlap, cudaStream_t stream) {
  using namespace f32;
  const Geom g = make_geom(nx, nz);
  const double len = direction == MW_DIR_X ? dx : dz;
  Args a{nx, nz, g.pitch, g.plane, d.hyc, d.hytc, d.hyi, d.hyti, d.hypi, d.srcw, d.in, d.out, d.s2, d.halo_in,
         d.halo_tmp, step_consts(len, dt_full, dt)};
  Device* dev = nullptr;
  int st = device(&dev);
  if (st) return st;
  const int sms = dev->sms.load(std::memory_order_relaxed);
  if (direction == MW_DIR_X) {
    // Cells per lane: 8 where the rows' runs then give every SM partition a
    // warp or more, else 4 (twice the warps, 9 instead of 5 % of them halo): a
    // few rows too long for the line kernels (us a step, eight a call, 4 / 8:
    // 20001x1 16.2 / 18.0, 20000x2 17.0 / 18.4, 16100x3 17.5 / 19.2, 16100x9 20.4 / 21.3).
    auto runs = [&](int v) { return (nx + x_run_max(v) - 1) / x_run_max(v); };
    const int v = (long long)runs(8) * nz >= 4LL * sms ? 8 : 4;
    const int nrun0 = runs(v), lenc = (nx + nrun0 - 1) / nrun0, nrun = (nx + lenc - 1) / lenc;
    const long long total = (long long)nrun * nz;
    const int resident = dev->x_ctas[v == 8] * sms;
    const unsigned grid = (unsigned)std::min<long long>(resident, (total + kXWarps - 1) / kXWarps);
    const size_t smem = (a.srcw ? (v == 8 ? sizeof(XBuf<8, true>) : sizeof(XBuf<4, true>))
                                : (v == 8 ? sizeof(XBuf<8>) : sizeof(XBuf<4>))) * 2 * kXWarps;
    auto kern = v == 8 ? (a.srcw ? k_dir_x_f32<8, true> : k_dir_x_f32<8, false>)
                       : (a.srcw ? k_dir_x_f32<4, true> : k_dir_x_f32<4, false>);
    return launch_overlapping(kern, dim3(grid), 32 * kXWarps, smem, stream, overlap, "FP32 x direction", a, nrun, lenc, total);
  }
  // Rows per z CTA: a CTA marches its tile and 12 rows more; an iteration takes
  // ~300 cycles alone on its SM and ~150 more for every CTA beyond two.
  const long long ncb = (nx + kZCols - 1) / kZCols;
  int tile = 1;
  double best = 0.0;
  for (int n = (nz + kZTileMax - 1) / kZTileMax; n <= std::max(1, nz / 8); n += std::max(1, n / 32)) {
    const int t = (nz + n - 1) / n;
    const long long ctas = ncb * ((nz + t - 1) / t);
    const long long per_sm = (ctas + sms - 1) / sms, waves = (per_sm + dev->z_ctas - 1) / dev->z_ctas;
    const double cost = (double)waves * (t + 12) * std::max(300.0, 150.0 * std::min<long long>(per_sm, dev->z_ctas));
    if (best == 0.0 || cost < best) {
      best = cost;
      tile = t;
    }
    if (t <= 8) break;
  }
  tile = (int)std::max<long long>(1, std::min<long long>(tile, (1LL << 32) / (4LL * g.pitch) - 24));  // >= 1: f32_dir_fits
  const int ntiles = (nz + tile - 1) / tile;
  for (int t0 = 0; t0 < ntiles; t0 += 65535) {
    const dim3 grid((unsigned)ncb, (unsigned)std::min(ntiles - t0, 65535));
    auto kern = a.srcw ? (a.s2 ? k_dir_z_f32<true, true> : k_dir_z_f32<true, false>)
                       : (a.s2 ? k_dir_z_f32<false, true> : k_dir_z_f32<false, false>);
    st = launch_overlapping(kern, grid, kZCols, z_smem(kZCols, tile, a.srcw != nullptr), stream,
                overlap && t0 == 0, "FP32 z direction", a, tile, t0);
    if (st) return st;
  }
  return MW_OK;
}

int launch_ens_f32(const EnsStageT<float>& es, int grid) {
  using namespace f32;
  if (es.n_items == 0) return MW_OK;
  Device* dev = nullptr;
  const int st = device(&dev);
  if (st) return st;
  if (es.direction == MW_DIR_X)
    k_ens_x_f32<<<grid, 32 * kXWarps, sizeof(XBuf<kEnsV>) * 2 * kXWarps, es.stream>>>(es);
  else
    (es.s2 ? k_ens_z_f32<true> : k_ens_z_f32<false>)<<<grid, kEnsZCols, z_smem(kEnsZCols, es.z_tile), es.stream>>>(es);
  return check_launch("ensemble FP32 direction launch");
}

int ens_f32_occupancy(int direction, int* blocks_per_sm) {
  using namespace f32;
  Device* dev = nullptr;
  const int st = device(&dev);
  if (st) return st;
  const cudaError_t e =
      direction == MW_DIR_X
          ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_ens_x_f32, 32 * kXWarps,
                                                          sizeof(XBuf<kEnsV>) * 2 * kXWarps)
          : cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k_ens_z_f32<false>, kEnsZCols,
                                                          z_smem(kEnsZCols, kEnsZTileMax));
  if (e != cudaSuccess) return fail(MW_ERR_CUDA, "occupancy query: %s", cudaGetErrorString(e));
  return MW_OK;
}

#if MW_CHECK
MW_OOB_COUNTER(oob_count_f32_dir)
#endif

}  // namespace mw
