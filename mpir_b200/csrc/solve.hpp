// Triangular-solve workspace and entry point (solve.cu).
#pragma once
#include <string>
#include <utility>

#include "engine.hpp"

namespace mpir {

struct SolveWorkspace {
  DeviceBuffer vals;      // the values that work items hand over (doubles): those
                          // of the forward solve, those of the backward; then
                          // the forward solve's result
  DeviceBuffer sync;      // tickets, one a direction
  DeviceBuffer err;       // SolveCtl: err = 1 when a bounded wait gave up, then
                          // the test controls of the waits (solve_dev.cuh)
  // Whether a direction's values are all marked pending (each direction's
  // launch marks the other's at its end).
  bool fwd_pending = false, bwd_pending = false;
  void allocate(const Plan &P);
  static size_t bytes_for(const Plan &P);
};

// Flags on the device, count of them stride apart: the full solve is left out
// when all are zero (p NULL: never).
struct ActiveFlags {
  const int32_t *p      = nullptr;
  int            count  = 0;
  int64_t        stride = 0;
};

// Phases of the solve, combinable as bits.
enum SolvePhase : int { kForward = 1, kDiagonal = 2, kBackward = 4, kAllPhases = 7 };

// x (permuted order, float64, device) <- (L D L^T)^{-1} x, or the phases
// selected: (L+I)^{-1} x, Dinv .* x, (L+I)^{-T} x (qdldl.hpp:362-432).
void ldlt_solve(const Plan &P, const Numeric &F, double *x, SolveWorkspace &ws,
                cudaStream_t s, int phases = kAllPhases, const ActiveFlags &act = ActiveFlags());

// Workspace of the several-vector solves (solve_multi.cu) for one width, as
// SolveWorkspace with nr values an entry.
struct MultiSolveWorkspace {
  int          nr = 0;  // vectors per application (4, 8 or 16)
  DeviceBuffer vals, sync, err;
  bool         fwd_pending = false;
  void         allocate(const Plan &P, int width);
  static size_t bytes_for(const Plan &P, int width);
};

// Vectors per several-vector application for nrhs right-hand sides (the
// kernels are instantiated for 4, 8 and 16; unused columns are zero).
int multi_width(int nrhs);

// X (n x width, column-major, leading dimension n, permuted order, float64,
// device) <- (L D L^T)^{-1} X, for all width columns at once (solve_multi.cu).
void ldlt_solve_multi(const Plan &P, const Numeric &F, double *X, int width,
                      MultiSolveWorkspace &ws, cudaStream_t s,
                      const ActiveFlags &act = ActiveFlags());

// QDLDL_solve (float32 factor, float64 x, host arrays) whose device data
// lives in a fixed file-scope array instead of allocated memory; see
// mpir_qdldl_solve_noalloc in include/mpir_b200.h.  Returns a status and a
// message in err.
int qdldl_solve_noalloc(int64_t n, const int64_t *Lp, const int64_t *Li, const float *Lx,
                        const float *Dinv, double *x, int device, std::string &err);

}  // namespace mpir
