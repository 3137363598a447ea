// Shared definitions for the B200 Krylov-Schur library (host and device).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "slepc_b200.h"

namespace b200 {

// Largest number of basis columns a BV may hold (ncv+1 plus the internal
// work column).  A Gram-Schmidt CTA holds 8 warps x 32 columns a lane, and a
// tile load's box has at most 256 columns.
constexpr int kMaxCols = 255;

// Number of spin iterations after which a device-side wait gives up.
constexpr long long kSpinLimit = 1ll << 22;

// Device error flags (bitmask written by kernels, read by the host).
enum DeviceError : int {
  kDevErrNone = 0,
  kDevErrInnerProduct = 1,   // BV_SafeSqrt rejected a negative inner product
  kDevErrTimeout = 2,        // a bounded wait (mbarrier / ticket) gave up
  kDevErrNonFinite = 4,      // NaN or Inf met in a reduction
};

// Gram-Schmidt pass actions (bitmask), decided on the device between passes.
enum GsAction : int {
  kActNone = 0,
  kActUpdate = 1,   // w <- w - V(:,0:j) coef
  kActDot = 2,      // partial dots V(:,0:j)^T w and w^T w
  kActScale = 4,    // w <- w * scale (normalisation)
};

// Stages of the DGKS state machine (what the pending dot result means).
enum GsStage : int {
  kStageDotOfPass = 0,     // c holds the dot of pass `pass`
  kStageExplicitNorm = 1,  // c holds V^T w' after pass `pass`; c[j] = ||w'||^2 gives the explicit norm
  kStageDone = 2,
};

// Per-BV device control block: the outcome of the last column orthogonalisation and the counters of
// the run it belongs to.  Written by the Gram-Schmidt kernel; the error bits stay until the host has
// read them and resets the block.
struct GsState {
  unsigned int ticket;  // word of the grid barrier (its top bit flips once per barrier)
  int lindep;           // linear dependence flag of the last finished column
  int halt;             // set when a Lanczos run broke down: later steps are skipped
  int halt_step;        // Lanczos step index at which the breakdown happened
  int err;              // DeviceError bits
  unsigned int run_ticket, run_exit;  // barrier and exit counters of a whole-run launch (zero between launches)
  int passes;           // passes done since the start of the run
  double beta_out;      // norm returned to the caller (BVOrthonormalizeColumn's norm)
  unsigned long long bytes;  // algorithmic bytes moved by those passes
};

}  // namespace b200

#define B200_CUDA_CHECK(expr)                                                         \
  do {                                                                                \
    cudaError_t _e = (expr);                                                          \
    if (_e != cudaSuccess) {                                                          \
      b200_set_last_error(__FILE__, __LINE__, cudaGetErrorString(_e));               \
      return B200_ERR_CUDA;                                                           \
    }                                                                                 \
  } while (0)

#define B200_CHECK(expr)                \
  do {                                  \
    b200_status _s = (expr);            \
    if (_s != B200_OK) return _s;       \
  } while (0)

#define B200_ARG_CHECK(cond, msg)                                 \
  do {                                                            \
    if (!(cond)) {                                                \
      b200_set_last_error(__FILE__, __LINE__, msg);               \
      return B200_ERR_ARG;                                        \
    }                                                             \
  } while (0)

extern "C" void b200_set_last_error(const char *file, int line, const char *msg);
