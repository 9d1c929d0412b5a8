// mw_fp64_line.cuh -- the line kernels' interface (mw_fp64_line.cu): one
// direction of a time step, all three RK stages, in one launch.
#pragma once

#include "mw_common.cuh"

namespace mw {

// Most cells of a grid that takes the line kernels: above this the CTAs of a
// launch come in several waves and the stage kernels, which need no whole lines
// in a CTA, do as well (us per step, eight a call, line kernels / six stage
// launches: 100x50 17.6 / 115, 300x150 41 / 116, 512x256 110 / 139, 800x400 236 / 272,
// 990x495 348 / 377; from half a million cells on it is one or the other by how
// the lines divide over the SMs: 880x620 400 / 384, 900x620 391 / 423, 1000x600
// 429 / 380, 1200x600 473 / 457).
constexpr long long kLineCellsMax = 600000;

// The double-FP32 form's (100x50 12.8 / 63, 300x150 18 / 74, 512x256 38 / 70, 700x500
// 85 / 109, 880x620 121 / 135; 600x1000 146 / 139, 1100x700 170 / 166, 1250x799
// 213 / 201).
constexpr long long kSplitLineCellsMax = 580000;
// Nor with lines of more cells than this, whose pieces (sixteen at most) take so
// many warps that an SM holds one or two CTAs (us a step, four a call, line
// kernels / six stage launches: 75x4000 90 / 107, 4000x120 127 / 125; 5000x100
// 154 / 138, 100x5000 166 / 144, 6000x75 141 / 123, 75x6000 148 / 128).
constexpr int kSplitLineMax = 4096;
// The FP32 form's against its direction kernels (40x12 8.7 / 19.1, 100x50 7.9 / 15.6,
// 300x150 8.7 / 16.6, 401x199 10.7 / 16.1, 512x256 12.5 / 19.1; 700x500 28.1 / 25.1,
// 1000x1000 61 / 40).  Grids of a few long rows lose earlier (four a call: 1500x200
// 31 / 26, 4000x75 39 / 26).
constexpr long long kF32LineCellsMax = 300000;

struct LineArgs {
  const double* hyc;
  const double* hytc;
  const double* hyi;
  const double* hyti;
  const double* hypi;
  const double* srcw;  // optional forcing of w
  const double* in;    // the direction's initial state
  double* out;         // its result; may be `in` where the lines are not cut (a CTA reads its lines before it writes them)
  double* s1;          // first and second stage, each optional
  double* s2;
  double* halo_in;     // optional: arrays that get the direction's halo of the initial state
  double* halo_tmp;    // and of the second stage
};

// How a direction's lines are spread over CTAs (fits where runs > 0): slots per lane, lines per CTA
// (log2), pieces per line and cells per piece, runs (warps) per line and cells
// per run, and a line's pitch in shared memory.
struct LineSpread {
  int sl = 0, log_lines = 0, pieces = 1, piece = 0, runs = 0, run = 0, lp = 0;
};

// Whether a grid takes the line kernels, and how.  cut: the lines of either
// direction are cut into pieces, so a direction's result must go to another
// array than its input.
struct LinePlan {
  LineSpread x, z;
  bool fits = false, cut = false;
};
int line_ieee_plan(int nx, int nz, LinePlan* plan);

// What the spread of a form's lines depends on.
struct LineKind {
  int min_slots;        // slots per lane, at least and at most (0: half a slot, the variables in two halves of a warp)
  int max_slots;
  int warps[3];         // most warps per CTA with none, one and two slots
  int regs[3];          // registers per thread with none, one and two slots
  int shared_slots;     // slots of a run that its neighbour has too
  int cell_bytes;       // shared memory per cell
  int row_bytes;        // and per cell of a column's row table (z)
  double tail;          // cost of a CTA's head and tail per warp (0: the IEEE form's rule)
};
inline size_t line_smem(const LineKind& kind, int lp, int log_lines, bool isx) {
  return ((size_t)lp * kind.cell_bytes << log_lines) + (isx ? 0 : (size_t)lp * kind.row_bytes);
}
LinePlan line_plan(const LineKind& kind, int nx, int nz, int sms);
int line_sms(int* out);  // SMs of the current device

// The same of the double-FP32 form (mw_split_line.cu).
int line_split_plan(int nx, int nz, LinePlan* plan);
int launch_line_split(const LinePlan& plan, int nx, int nz, double dx, double dz, double dt_full, double dt,
                      const LineArgs& a, int direction, bool overlap, cudaStream_t stream);

// One direction of one step of size dt.  overlap: the kernel may start while
// the one before it on the stream is finishing, and waits for it before it
// touches the state; only for a launch behind another line kernel of the same
// call (what it reads before the wait, the backgrounds, is then complete).
int launch_line_ieee(const LinePlan& plan, int nx, int nz, double dx, double dz, double dt_full, double dt,
                     const LineArgs& a, int direction, bool overlap, cudaStream_t stream);

// The plan of a form that has line kernels (else one that fits no grid).
inline int line_plan_of(int f64_mode, int nx, int nz, LinePlan* plan) {
  *plan = LinePlan();
  return f64_mode == MW_F64_IEEE ? line_ieee_plan(nx, nz, plan)
                                 : (f64_mode == MW_F64_SPLIT ? line_split_plan(nx, nz, plan) : MW_OK);
}

}  // namespace mw
