// mw_f32_dir.cuh -- the FP32 direction kernels' interface (mw_f32_dir.cu).
#pragma once

#include "mw_common.cuh"

namespace mw {

struct F32DirArgs {
  const double* hyc;
  const double* hytc;
  const double* hyi;
  const double* hyti;
  const double* hypi;
  const double* srcw;  // optional forcing of w
  const float* in;     // the direction's initial state
  float* out;          // its result; must not overlap `in` (launch_dir_f32)
  float* s2;           // second stage (optional)
  float* halo_in;      // optional: arrays that get the direction's halo of the initial state
  float* halo_tmp;     // and of the second stage
};

// HV = -2 hv of the FP32 form (hv = -hv_beta d / (16 dt_full)) and the update's
// factor dt_stage / (2 d): the kernels carry values and fluxes times 2.
inline float f32_hv(double d, double dt_full) { return (float)(2.0 * kHvBeta * d / (16 * dt_full)); }
inline float f32_c(double d, double dt_stage) { return (float)(dt_stage / (2.0 * d)); }

// Whether a row is short enough for the z pass's 32-bit offsets within a tile
// (25 rows below 2^32 bytes); longer ones are stepped stage by stage.
inline bool f32_dir_fits(int nx) { return 25LL * 4 * (nx + 4LL) < (1LL << 32); }

// One direction of one step of size dt; overlap as for the line kernels
// (mw_fp64_line.cuh).
int launch_dir_f32(int nx, int nz, double dx, double dz, double dt_full, double dt, const F32DirArgs& d, int direction,
                   bool overlap, cudaStream_t stream);

// The same by line kernels (mw_f32_line.cu), for grids whose lines fit a CTA;
// `out` may be `in` where the plan does not cut the lines.
struct LinePlan;
int line_f32_plan(int nx, int nz, LinePlan* plan);
int launch_line_f32(const LinePlan& plan, int nx, int nz, double dx, double dz, double dt_full, double dt,
                    const F32DirArgs& d, int direction, bool overlap, cudaStream_t stream);

}  // namespace mw
