// mw_line.cuh -- what the line kernels of the IEEE-FP64 (mw_fp64_line.cu) and
// double-FP32 (mw_split_line.cu) forms share: which cells a CTA holds, and the
// passes over them between global and shared memory.
#pragma once

#include "mw_common.cuh"
#include "mw_fp64_line.cuh"

namespace mw {
namespace {

constexpr int kLineMax = 8;            // most lines per CTA
constexpr size_t kLineSmem = 200 << 10;
// A launch of at most this many CTAs, about one per SM, lets the next one in at
// its head, whose row constants then cost no time (us a step, eight in a call:
// IEEE form 60x30 17.9 -> 16.6, 100x50 18.2 -> 17.6, 150x75 21.7 -> 20.5, double-FP32
// 100x50 14.2 -> 12.8); a larger one only after its last stage: the next one's CTAs
// take what is free beside its own, and earlier that is unevenly much (IEEE,
// 256x128: 47.6 us a step with the trigger at the head, 37.9 here; 300x150 57, 41).
constexpr unsigned kLineFewCtas = 152;

struct LineShape {
  int n, nlines;         // cells per line, lines
  int log_lines, runs;   // lines per CTA (a power of two), runs per line
  int run;               // cells per run
  int pieces, piece;     // pieces per line, cells per piece
  int lp;                // shared-memory pitch of a line
  int pitch;
  long long plane;
};
struct LineGeom : LineShape {
  LineArgs a;
};

// The shape of a direction's launch, its CTAs and threads per CTA.
inline void set_line_geom(LineShape* P, const LineSpread& sp, int nx, int nz, bool isx, int* ctas, int* threads) {
  const Geom g = make_geom(nx, nz);
  P->n = isx ? nx : nz;
  P->nlines = isx ? nz : nx;
  P->pitch = g.pitch;
  P->plane = g.plane;
  P->log_lines = sp.log_lines;
  P->pieces = sp.pieces;
  P->piece = sp.piece;
  P->run = sp.run;
  P->runs = sp.runs;
  P->lp = sp.lp;
  *threads = 32 * (sp.runs << sp.log_lines);
  *ctas = ((P->nlines + (1 << sp.log_lines) - 1) >> sp.log_lines) * sp.pieces;
}

#define MW_LG(p, off) MW_AT((p), (off), 4 * P.plane)

// The halo cells that cell c of a line is the source of, in a global array; v[0 .. NV): variables q0 onwards.
template <int DIR, int NV = 4>
__device__ __forceinline__ void halo_out(const LineGeom& P, double* g, int line, int c, const double* v,
                                         const double* hr, int q0 = 0) {
  const int n = P.n;
  if (DIR == MW_DIR_X) {
    const long long row = (long long)(line + kHs) * P.pitch;
    for (int q = q0; q < q0 + NV; ++q) {
      if (c < kHs) MW_LG(g, q * P.plane + row + n + kHs + c) = v[q - q0];
      if (c >= n - kHs) MW_LG(g, q * P.plane + row + c - n + kHs) = v[q - q0];
    }
  } else {
    for (int q = q0; q < q0 + NV; ++q)
      for (int h = 0; h < 4; ++h)
        if (c == (h < 2 ? 0 : n - 1))
          MW_LG(g, q * P.plane + (long long)(h < 2 ? h : n + h) * P.pitch + line) =
              q == WMOM ? 0.0 : (q == UMOM ? v[q - q0] * hr[h] : v[q - q0]);
  }
}

// Cells [ca, cb) of the CTA's lines, each by one thread: fn(line, cell, offset in a plane of a global array).
template <int DIR, typename Fn>
__device__ __forceinline__ void each_cell4(const LineShape& P, int l0, int nl, int ca, int cb, Fn fn) {
  const int len = cb - ca;
  for (int i = threadIdx.x; i < (DIR == MW_DIR_X ? len * nl : len << P.log_lines); i += blockDim.x) {
    int l, c;
    if (DIR == MW_DIR_X) {
      l = i / len;
      c = ca + i - l * len;
    } else {
      l = i & ((1 << P.log_lines) - 1);
      c = ca + (i >> P.log_lines);
      if (l >= nl) continue;
    }
    const int cw = DIR == MW_DIR_Z ? c : (c < 0 ? c + P.n : (c >= P.n ? c - P.n : c));
    fn(l, c, DIR == MW_DIR_X ? (long long)(l0 + l + kHs) * P.pitch + kHs + cw
                             : (long long)(cw + kHs) * P.pitch + l0 + l + kHs);
  }
}

// The four x-halo columns of the wall halo rows, from the halo columns' own first and last rows (8 threads).
__device__ __forceinline__ void halo_corners(const LineGeom& P, const double* hr) {
  const LineArgs& a = P.a;
  const int n = P.n;
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

}  // namespace
}  // namespace mw
