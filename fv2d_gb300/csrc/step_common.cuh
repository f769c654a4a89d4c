// step_common.cuh -- data structures shared by the host API and the FP64
// kernels of the plain (drop-in) path.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace fv2d {

constexpr int HALO = 2; // ghost depth read by PLM + the 3x3 viscous stencil

// Tile of interior cells owned by one CTA of the fused step kernel.
template <int TX_, int TY_, int NT_>
struct Tile {
  static constexpr int TX = TX_;             // cells along x (even: TMA rows start on 16-byte boundaries)
  static constexpr int TY = TY_;             // cells along y
  static constexpr int SW = TX + 2 * HALO;   // staged tile width  (TMA box x)
  static constexpr int SH = TY + 2 * HALO;   // staged tile height (TMA box y)
  static constexpr int NT = NT_;             // threads per CTA
};
using WideTile = Tile<16, 16, 288>;  // 9 warps: the 544 faces of a tile in two rounds
using SmallTile = Tile<8, 8, 160>;   // 5 warps: the 144 faces of a tile in one round
enum { TILE_WIDE = 0, TILE_SMALL = 1 };

enum { RECON_PCM = 0, RECON_PLM = 2, RECON_MH = 3 };
enum { STAGE_EULER = 0, STAGE_RK2_PREDICT = 1, STAGE_RK2_CORRECT = 2 };
enum { RUN_RUNNING = 0, RUN_DONE = 1, RUN_SAVE = 2, RUN_NUMERIC = 3, RUN_PAUSED = 4 };
enum { DEVERR_TMA_TIMEOUT = 1, DEVERR_BOUNDS = 2 };

// The simulation clock: what a committed step leaves behind.
struct Clock {
  double t;          // time after the last committed update (main.cpp:83)
  double dt;         // CFL dt of the current primitive state (ComputeDt.h:64)
  double inv_hyp;    // max inverse hyperbolic dt of the current state
  double last_dt;    // dt used by the last update
  unsigned long long counters[3];  // checkNegatives counts of the last update
  int parity;        // which primitive buffer holds the current state
  int ite;           // committed updates
  int status;        // RUN_*
  int steps_in_call; // iterations done by the current fv2d_advance
};

// Reductions of a step that is not committed yet.
struct StepSums {
  unsigned long long hyp;  // running max of the inverse hyperbolic dt (bits of a non-negative double)
  unsigned long long cnt[3];
};

// Clock, reductions and loop control, resident in device memory.  Between
// calls clock[0] is the state and every StepSums is zero.  A step followed by
// commit_kernel reduces into pending[0], which that kernel commits to clock[0].
// In a chained sequence (StepArgs::chained) step k commits step k - 1 itself: its
// CTAs all form the new clock from clock[k & 1] and pending[(k - 1) & 3], one
// of them stores it in clock[(k + 1) & 1] and clears pending[(k + 1) & 3] (last
// read two launches ago), and they reduce into pending[k & 3]; commit_kernel
// ends the sequence.  No launch writes what another CTA of it reads.
struct DevState {
  Clock clock[2];
  StepSums pending[4];
  double tend, next_save, eps;  // device-driven loop control
  double one;        // 1.0 (Adder, physics.cuh)
  int check_save;    // stop before an iteration that must write a snapshot
  int max_steps;     // iteration cap of the current fv2d_advance
  int log_cap;       // capacity of the per-iteration log (records)
  int error;         // DEVERR_* bit set by a kernel that gave up waiting
  unsigned int ticket;  // CTAs of the set-up pass that finished
  int pad;
};

// Constants of the binary32 bound on a cell's inverse dt (physics.cuh).
struct DtBound {
  float gamma, inv_dx, inv_dy;  // NaN: no bound, every cell is evaluated
};

// Everything one step launch needs besides the two tensor maps.
struct StepArgs {
  double *Q[2];       // primitive planes (4 planes, ghosts included)
  double *U;          // conservative planes (same layout)
  double *U1;         // RK2 predictor planes (same layout)
  const float *grav_row;  // analytical gravity per interior row (float, Gravity.h:16)
  const double *kap_row;  // per interior row: kappaL, kappaR, kappaU, kappaD
  DevState *st;
  double *log;        // per-iteration records {t, dt, inv_hyp, 3 counters} (may be null)
  long long plane;    // elements per field plane
  int pitch;          // elements per padded row
  int Nx, Ny;
  int nblocks;
  int stage;          // STAGE_*
  int driven;         // 1: dt and loop control from DevState
  int chained;        // 1: step `step` of a sequence that commits its own steps
  int step;
  int overlapped;     // 1: dispatched while the previous launch runs
  double dt_arg;      // dt when driven == 0
  // gas and mesh constants
  double gamma, gm1, entho, fslp_K;
  double dx, dy, inv_dx, inv_dy;
  int dx_pow2, dy_pow2;  // 1/dx (1/dy) is exact: divisions become products
  uint32_t rw_dx, rw_dy;  // otherwise quotients by dx (dy) share its reciprocal word
  double one_over_dx, one_over_dy;  // 1.0/dx, 1.0/dy (Viscosity.h:57-58)
  double gx_dx, gy_dy;  // FSLP gravity terms gx*dx, gy*dy (Update.h:119)
  double gxf, gyf;      // constant gravity narrowed to float (Gravity.h:39)
  double eps_reset;     // epsilon_reset_negative
  double CFL, inv_tc, inv_visc;  // dt finalisation (ComputeDt.h:64)
  DtBound bound;  // binary32 bound of a cell's inverse dt
  double mu;
  double bctc_ymin_value, bctc_ymax_value;
  int bcx, bcy;
  int grav_mode;  // 0 none, 1 constant, 2 analytical
  int tc, visc, wb;
  int bctc_ymin, bctc_ymax;
  double *mirror;  // device view of a page-locked host (Ny x Nx x 4) array that the
                   // final stage also writes the new primitives to (may be null)
};

// Set-up pass arguments (interior upload -> planes, ghosts, U, dt reduction).
struct PrepArgs {
  const double *q_aos;  // interior primitives, interleaved (Ny x Nx x 4)
  double *Q;            // destination primitive planes (current buffer)
  double *U;
  DevState *st;
  long long plane;
  int pitch, Nx, Ny, nblocks;
  double gamma, gm1, dx, dy, inv_dx, inv_dy;
  int dx_pow2, dy_pow2;
  uint32_t rw_dx, rw_dy;
  double CFL, inv_tc, inv_visc;
  DtBound bound;
  int bcx, bcy;
};

}  // namespace fv2d
