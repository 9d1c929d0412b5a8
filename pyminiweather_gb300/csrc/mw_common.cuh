// mw_common.cuh -- constants, host-side argument checks and error plumbing
// shared by the translation units of libminiweather_gb300.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>

#include "../../include/miniweather_gb300.h"

// MW_CHECK=1 builds the bounds-checked library (a debug build): the kernels
// that access memory through MW_AT count every index outside its array
// instead of touching memory there, and mw_debug_oob_count reads the count.
#ifndef MW_CHECK
#define MW_CHECK 0
#endif

namespace mw {

#if MW_CHECK
static __device__ unsigned long long g_oob_count;           // per translation unit
static __device__ __align__(16) unsigned char g_oob_sink[128];  // stands in for out-of-range elements

template <typename T, typename I>
__device__ __forceinline__ T& checked_at(T* p, I i, long long n) {
  static_assert(sizeof(T) <= sizeof(g_oob_sink), "element larger than the sink");
  if ((long long)i < 0 || (long long)i >= n) {
    atomicAdd(&g_oob_count, 1ULL);
    return *reinterpret_cast<T*>(g_oob_sink);
  }
  return p[i];
}
#define MW_AT(p, i, n) (::mw::checked_at((p), (i), (long long)(n)))
// Adds this translation unit's count to *out (and resets it).
#define MW_OOB_COUNTER(fn)                                                          \
  int fn(unsigned long long* out, bool reset) {                                     \
    unsigned long long v = 0;                                                       \
    cudaError_t e = cudaMemcpyFromSymbol(&v, g_oob_count, sizeof(v));               \
    if (e == cudaSuccess && reset) {                                                \
      const unsigned long long z = 0;                                               \
      e = cudaMemcpyToSymbol(g_oob_count, &z, sizeof(z));                           \
    }                                                                               \
    if (e != cudaSuccess) return fail(MW_ERR_CUDA, "oob counter: %s", cudaGetErrorString(e)); \
    *out += v;                                                                      \
    return MW_OK;                                                                   \
  }
#else
#define MW_AT(p, i, n) ((p)[(i)])
#endif

// Physical constants, pyminiweather/data/constants.py:13-27.
constexpr double kHvBeta = 0.05;
constexpr double kP0 = 1.0e5;
constexpr double kC0 = 27.5629410929725921310572974482;
constexpr double kGamma = 1.40027894002789400278940027894;
constexpr double kGrav = 9.8;
constexpr double kCp = 1004.0;
constexpr double kCv = 717.0;
constexpr double kRd = 287.0;
constexpr double kPi = 3.14159265358979323846264338327;
constexpr double kTheta0 = 300.0;
constexpr double kExner0 = 1.0;

constexpr int kHs = 2;  // halo width (params["hs"], fixed at 2 by the reference CLI)
enum { DENS = 0, UMOM = 1, WMOM = 2, RHOT = 3 };

// Geometry of one (4, nz+4, nx+4) state array.
struct Geom {
  int nx, nz;
  int pitch;          // nx + 4
  long long plane;    // (nz + 4) * (nx + 4)
};

inline Geom make_geom(int nx, int nz) {
  Geom g;
  g.nx = nx;
  g.nz = nz;
  g.pitch = nx + 2 * kHs;
  g.plane = (long long)(nz + 2 * kHs) * (nx + 2 * kHs);
  return g;
}

// ---------------------------------------------------------------------------
// Host-side error state (one message per calling thread).
void set_error(const char* fmt, ...);
int fail(int code, const char* fmt, ...);
int check_launch(const char* what);

inline bool finite_pos(double v) { return std::isfinite(v) && v > 0.0; }

template <typename T>
inline bool aligned(const T* p) {
  return ((uintptr_t)p % alignof(T)) == 0;
}

inline bool ranges_overlap(const void* a, size_t abytes, const void* b, size_t bbytes) {
  uintptr_t a0 = (uintptr_t)a, b0 = (uintptr_t)b;
  return a0 < b0 + bbytes && b0 < a0 + abytes;
}

int check_grid(int nx, int nz);

// HV = -12 hv of the IEEE-FP64 form (hv = -hv_beta d / (16 dt_full),
// interpolate.py:101,149), whose kernels carry fluxes divided by it: held above
// 2^-400 (dt_full / d above 2^395), where the hyperviscosity term is far below
// rounding either way.
inline double ieee_hv(double d, double dt_full) { return std::fmax(12.0 * kHvBeta * d / (16 * dt_full), 0x1p-400); }

// The scale of a direction's fluxes in that form and the factor of its update,
// c = HV dt / (12 d).  What is advected takes part as c / HV: mass as c IHV, the
// rest as c over H12 (times rho) or c I12 (pressure), each twelve times rounded
// numbers whose error stays the same over a run and makes every flux too large or
// too small by it.  So of the numbers next to HV (within 16 ulps; the
// hyperviscosity, a small part of a flux, is that much off) the one is taken for
// which the three products are closest to dt / d: 0.25 x 2^-53 off on average over
// the grids of the tests and the timing cases, 0.5 with dt / (12 d) as the only
// rounded number, 0.8 with HV as it comes.  rel-L2 errors of rho' and (rho theta)'
// by stages, against 64-bit significands, as chosen / HV as it comes: 200 steps at
// 200x100 2.4e-15 / 3.5e-15 and 1.2e-15 / 2.8e-15; 300 at 100x50 1.35e-14 / 1.57e-14
// and 4.1e-15 / 10.1e-15.
struct IeeeScale {
  double HV, IHV, H12, I12, c;
};
inline IeeeScale ieee_scale(double d, double dt_full, double dt) {
  auto at = [&](double hv) {
    IeeeScale s;
    s.HV = hv;
    s.IHV = 1.0 / hv;
    s.H12 = 12.0 * hv;
    s.I12 = 12.0 * s.IHV;
    s.c = dt / (12.0 * d) * hv;
    return s;
  };
  const double hv0 = ieee_hv(d, dt_full);
  IeeeScale best = at(hv0);
  // t = dt / (12 d) to twice the precision, th + tl
  const double e = 12.0 * d, el = std::fma(12.0, d, -e), th = dt / e, rth = 1.0 / th;
  const double tl = (std::fma(-th, e, dt) - th * el) / e;
  const double big = std::fmax(std::fabs(th), std::fabs(best.c)), small = std::fmin(std::fabs(th), std::fabs(best.c));
  if (!(small > 0x1p-400 && big < 0x1p400 && hv0 < 0x1p400 && hv0 > 0x1p-400)) return best;  // products out of range
  double least = 1.0;
  long long bits;
  std::memcpy(&bits, &hv0, sizeof bits);
  for (int k = 0; k <= 32; ++k) {  // hv0, then outwards
    const long long b = bits + (k & 1 ? (k + 1) / 2 : -(k / 2));
    double hv;
    std::memcpy(&hv, &b, sizeof hv);
    IeeeScale s = at(hv);
    s.c = std::fma(tl, hv, th * hv);
    // relative errors of c IHV, 12 c / H12 and c I12 / 12
    auto off = [&](double x, double y, double f) {  // x y - f t, over f t (f: 1 or 12)
      const double p = x * y, q = f * th;
      return ((p - q) + (std::fma(x, y, -p) - (std::fma(f, th, -q) + f * tl))) * rth / f;
    };
    const double p = 12.0 * s.c, q = th * s.H12;
    const double e1 = ((p - q) + (std::fma(12.0, s.c, -p) - (std::fma(th, s.H12, -q) + tl * s.H12))) / q;
    const double worst = std::fmax(std::fmax(std::fabs(off(s.c, s.IHV, 1.0)), std::fabs(e1)),
                                   std::fabs(off(s.c, s.I12, 12.0)));
    if (worst < least) {
      least = worst;
      best = s;
    }
  }
  return best;
}

inline bool valid_f64_mode(int m) { return m == MW_F64_NATIVE || m == MW_F64_SPLIT || m == MW_F64_IEEE; }

// Internal launch flag: the launch may start while the one before it on the
// stream is finishing (programmatic dependence).  Only behind another launch of
// the same call: what a kernel reads before overlap_wait(), the backgrounds, is
// then complete.  Never taken from a caller's flags (user_flags).
constexpr unsigned kFlagOverlap = 1u << 31;
inline unsigned user_flags(unsigned flags) { return flags & ~kFlagOverlap; }

#ifdef __CUDACC__
// Before anything the launch before may have written is touched (no effect in a plain launch).
__device__ __forceinline__ void overlap_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The next launch may come in, once every CTA of this one has got here or ended.
// Not called early in a kernel whose CTAs do not fill the SMs evenly: the next
// one's CTAs take what is free beside them, and stay where that was (FP64 stage
// launches at 992x992, called at the head: 911 us a step, not at all: 643, plain
// launches 657).
__device__ __forceinline__ void overlap_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Zeroes the halo cells of a (4, nz+4, nx+4) array: the two halo rows at either end, contiguous, and the four halo
// columns of the rows between, over all threads of the launch.  (A CTA to a row: a stage adjoint at 3000000x2, whose
// halo is mostly four long rows, 1640 us against 420.)
template <typename T>
__device__ __forceinline__ void zero_frame(T* g, int nx, int nz, long long plane) {
  const long long pitch = nx + 2 * kHs, span = kHs * pitch, step = (long long)gridDim.x * blockDim.x;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  auto zero = [&](long long o) {
#pragma unroll
    for (int q = 0; q < 4; ++q) MW_AT(g, q * plane + o, 4 * plane) = T(0);
  };
  for (long long e = t; e < 2 * span; e += step) zero(e < span ? e : plane - 2 * span + e);
  for (long long e = t; e < 2LL * kHs * nz; e += step) {
    const int h = (int)e & (2 * kHs - 1);
    zero((e / (2 * kHs) + kHs) * pitch + (h < kHs ? h : nx + h));
  }
}

template <typename... P, typename... A>
int launch_overlapping(void (*kernel)(P...), dim3 grid, int threads, size_t smem, cudaStream_t stream, bool overlap,
                       const char* what, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = overlap ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, P(args)...);
  return e == cudaSuccess ? MW_OK : fail(MW_ERR_CUDA, "%s launch: %s", what, cudaGetErrorString(e));
}
#endif

// Rows per z CTA for a single-grid launch: the largest tile up to max_rows
// that still gives about two CTAs per SM (152 SMs), at least 8 rows.
inline int z_tile_rows(int nx, int nz, int cols_per_cta, int max_rows) {
  const long long ncb = (nx + cols_per_cta - 1) / cols_per_cta;
  long long t = (long long)nz * ncb / 304;
  if (t > max_rows) t = max_rows;
  if (t < 8) t = 8;
  return (int)t;
}

}  // namespace mw

#define MW_REQUIRE(cond, code, ...)            \
  do {                                         \
    if (!(cond)) return mw::fail((code), __VA_ARGS__); \
  } while (0)
