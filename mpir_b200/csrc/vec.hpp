// Vector operations of the GMRES-IR loop (vec.cu).
#pragma once
#include <cstdint>
#include <cstring>

#include "engine.hpp"

namespace mpir {

// Owns the max-norm slots of one solver, eight a vector, read back with
// read_inf: 0 residual, 1 |d|, 2 |x_old|, 3 |b_scaled|, 4..7 backward-error
// terms.  The forms with nb take that many vectors n apart (bit k of act:
// vector k takes part); per vector the arithmetic is that of one vector.
class VecOps {
 public:
  int64_t      n = 0;
  DeviceBuffer infbits;
  int          batch = 1;  // vectors a call may take at once

  void allocate(int64_t n, int batch = 1);
  void spmv(int nb, const int64_t *Kp, const int32_t *Kj, const double *Kv, const double *x, double *y,
            cudaStream_t s);
  // clear: slot 0 is zeroed first (else something before has).
  void residual(int nb, uint32_t act, const int64_t *Kp, const int32_t *Kj, const double *Kv,
                const double *x, const double *b, double *r, bool dd, bool clear, cudaStream_t s);
  void backward_terms(int nb, const int64_t *Kp, const int32_t *Kj, const double *Korig,
                      const double *x, const double *ADp, const double *bp, cudaStream_t s);
  void scale(const double *x, double a, double *y, cudaStream_t s);
  // d *= scale, x += d; infinity norms of d and of the old x (each entry
  // times w[i] when w is given: the norms of the unscaled vectors).
  void ir_update(double *d, double scale, double *x, cudaStream_t s,
                 const double *w = nullptr);
  // x <- x rounded to the factor's storage type (1 float32, 2 bfloat16,
  // 3 float16; float64 leaves x unchanged).
  void round_to(int prec, double *x, cudaStream_t s);
  void rhs_in(int nb, const int64_t *perm, const double *AD, const double *b, double *bs,
              double *ADp, double *bp, cudaStream_t s);
  void sol_out(int nb, const int64_t *perm, const double *ADp, const double *x, double *out,
               cudaStream_t s);
  // All 8 slots of vectors 0 .. nb-1 into h[8 k + slot].
  void read_inf(int nb, double *h, cudaStream_t s);
};

}  // namespace mpir
