// Device side of PrecondGmres (gmres_ir.hpp:636-741): arnoldi.cu.
#pragma once
#include <algorithm>
#include <cstdint>

#include "engine.hpp"

namespace mpir {

constexpr int kMaxVectors = 16;  // vectors a call takes in lockstep

// Factors and flags of up to kMaxVectors vectors, passed by value.
struct VecFactors {
  double v[kMaxVectors];
};

// Per-vector state in device memory.
struct GmresCtl {
  double  rho;      // residual norm of the least-squares problem
  int32_t k;        // basis vectors so far
  int32_t active;   // the next step is taken
  int32_t reorth;   // columns orthogonalised twice
  int32_t began;    // rho of the right-hand side was not below tol
  int32_t pad[2];
};
// What the host reads: written by the kernels to pinned host memory.
struct GmresMail {
  int32_t active[2][kMaxVectors];  // after a step, by the step's parity
  int32_t k[kMaxVectors], reorth[kMaxVectors], began[kMaxVectors];
};

// The state of the vectors of a call: control words, the triangular factor R
// of the Hessenberg matrix (column j's j + 1 entries at j (j + 1) / 2), the
// rotations, their right-hand side and the solution of the least-squares
// problem.  It is laid out for kSteps steps at first and grows with the steps that
// are taken: a caller that allows n of them, as many as there can be, would have
// n^2 / 2 values of R reserved.
class Arnoldi {
 public:
  void   allocate(int64_t n, int64_t m, int vectors);
  size_t bytes() const { return state_.bytes() + wide_.bytes(); }
  static constexpr int64_t kSteps = 512;
  // Bytes at first.
  static size_t bytes_for(int64_t m, int vectors) {
    return stride(std::min(m, kSteps)) * vectors * sizeof(double);
  }
  ~Arnoldi();
  Arnoldi() = default;
  Arnoldi(const Arnoldi &)            = delete;
  Arnoldi &operator=(const Arnoldi &) = delete;

  // Vector k of every block at k * n; bit k of act: vector k takes part.
  // Steps there is room for, and room for more (waits for the stream; the flags move).
  int64_t room() const { return cap_; }
  void    reserve(int nb, int64_t steps, cudaStream_t s);
  // begin:  V_0 = b fac, its norm against tol.
  void begin(int nb, uint32_t act, const double *b, const VecFactors &fac, double *V, double tol,
             cudaStream_t s);
  // first:  after the preconditioner, V_0 /= |V_0|.
  void first(int nb, double *V, double tol, cudaStream_t s);
  // step j: w = V_{j+1} (preconditioned) made orthogonal to V_0 .. V_j, its
  // column of H, the rotations, whether to go on (mail().active[j % 2]).
  void step(int nb, int64_t j, double *V, int64_t block, double tol, cudaStream_t s);
  // end:    d = sum y_j V_j for the vectors of act; x = d, or (update)
  // x += d scale with max |d scale| and max |x before| into inf[8 k + 1],
  // inf[8 k + 2] and zero into inf[8 k].
  void end(int nb, uint32_t act, const double *V, int64_t block, double *x, bool update,
           const VecFactors &scale, unsigned long long *inf, cudaStream_t s);

  const GmresMail &mail() const { return *mail_; }
  // Active flags on the device (int32, active_stride() apart) for kernels that
  // are skipped when no vector is active.
  const int32_t *active() const;
  int64_t        active_stride() const { return stride(cap_) * 2; }

 private:
  static int64_t stride(int64_t m) {
    return (4 + m * (m + 1) / 2 + 2 * m + (m + 1) + m + (m + 2) + 1) / 2 * 2;
  }
  int          cluster() const;
  bool         wide(int nb) const;  // swept by the whole chip
  int64_t      n_ = 0, m_ = 0, cap_ = 0;  // steps allowed, laid out
  int          vectors_ = 0;
  DeviceBuffer state_, wide_;
  GmresMail   *mail_ = nullptr;
};

}  // namespace mpir
