// Vector kernels around the GMRES steps (arnoldi.cu): the symmetric SpMV and
// residual in float64 or double-double (MatrixMultiply / VectorSubtract,
// ops.hpp:25-96), max-norms (InfNrm, ops.hpp:300-329), the gather and scatter
// between the caller's order and the factor's, and the update of plain
// refinement.
#include <cfloat>
#include <cmath>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "vec.hpp"

namespace mpir {

// ---------------------------------------------------------------------------
// Double-double helpers (Knuth's TwoSum and the FMA form of Dekker's
// TwoProduct): a value is the unevaluated sum hi + lo.
struct dd {
  double hi, lo;
};
__device__ __forceinline__ dd two_sum(double a, double b) {
  const double s  = a + b;
  const double bb = s - a;
  const double e  = (a - (s - bb)) + (b - bb);
  return {s, e};
}
__device__ __forceinline__ dd quick_two_sum(double a, double b) {
  const double s = a + b;
  return {s, b - (s - a)};
}
__device__ __forceinline__ dd two_prod(double a, double b) {
  const double p = a * b;
  return {p, fma(a, b, -p)};
}
__device__ __forceinline__ dd dd_add(dd a, dd b) {
  dd s = two_sum(a.hi, b.hi);
  dd t = two_sum(a.lo, b.lo);
  s.lo += t.hi;
  s = quick_two_sum(s.hi, s.lo);
  s.lo += t.lo;
  return quick_two_sum(s.hi, s.lo);
}

__device__ __forceinline__ void atomic_max_abs(unsigned long long *slot, double v) {
  atomicMax(slot, static_cast<unsigned long long>(__double_as_longlong(fabs(v))));
}

// Max of |v| over the warp, then one atomic per warp.  The maximum is taken
// on the bit patterns of |v| (non-negative doubles order as their bits), so a
// NaN (whose |v| pattern lies above infinity's) wins and is reported: fmax
// would drop it and a non-finite residual would pass for a small one.
__device__ __forceinline__ void warp_max_abs(unsigned long long *slot, double v,
                                             bool active) {
  unsigned long long a =
      active ? static_cast<unsigned long long>(__double_as_longlong(fabs(v))) : 0ull;
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long b = __shfl_xor_sync(0xffffffffu, a, o);
    a                          = b > a ? b : a;
  }
  if ((threadIdx.x & 31) == 0) atomicMax(slot, a);
}

// ---------------------------------------------------------------------------
// SpMV with G lanes per row over the full symmetric CSR.
//   MODE 0: y = K x
//   MODE 1: y = b - K x,           max|y| into inf[0]
//   MODE 2: y = b - K x in double-double, rounded to float64, max into inf[0]
//
// Batched form (all kernels below): blockIdx.y selects vector k of a batch,
// the vectors k*vs apart, its max-norm slots at inf + 8k, and k is skipped
// unless bit k of vact is set.  One vector is gridDim.y == 1.
__device__ __forceinline__ bool batch_skip(uint32_t vact) { return !(vact >> blockIdx.y & 1u); }

template <int G, int MODE>
__global__ void k_spmv(int64_t n, const int64_t *Kp, const int32_t *Kj,
                       const double *Kv, const double *x, const double *b,
                       double *y, unsigned long long *inf, int64_t vs,
                       uint32_t vact) {
  grid_wait();
  if (batch_skip(vact)) return;
  x += blockIdx.y * vs;
  y += blockIdx.y * vs;
  if (b) b += blockIdx.y * vs;
  if (inf) inf += 8 * blockIdx.y;
  const int64_t gid  = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t row  = gid / G;
  const int     lane = threadIdx.x % G;
  const bool    act  = row < n;
  if (MODE == 2) {
    dd s{0.0, 0.0};
    if (act)
      for (int64_t e = Kp[row] + lane; e < Kp[row + 1]; e += G)
        s = dd_add(s, two_prod(Kv[e], x[Kj[e]]));
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      dd t{__shfl_xor_sync(0xffffffffu, s.hi, o, G),
           __shfl_xor_sync(0xffffffffu, s.lo, o, G)};
      s = dd_add(s, t);
    }
    double r = 0.0;
    if (act && lane == 0) {
      dd rr = dd_add(dd{b[row], 0.0}, dd{-s.hi, -s.lo});
      r     = rr.hi + rr.lo;
      y[row] = r;
    }
    warp_max_abs(inf, r, act && lane == 0);
    return;
  }
  double s = 0.0;
  if (act)
    for (int64_t e = Kp[row] + lane; e < Kp[row + 1]; e += G) s += Kv[e] * x[Kj[e]];
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, G);
  if (MODE == 0) {
    if (act && lane == 0) y[row] = s;
  } else {
    double r = 0.0;
    if (act && lane == 0) {
      r      = b[row] - s;
      y[row] = r;
    }
    warp_max_abs(inf, r, act && lane == 0);
  }
}

// Backward-error terms on the original (unscaled) system in permuted order:
// inf = {max|b - K xo|, max_i sum_j |k_ij|, max|xo|, max|b|}, where
// xo = x .* ADp.
template <int G>
__global__ void k_backward_terms(int64_t n, const int64_t *Kp, const int32_t *Kj,
                                 const double *Korig, const double *x,
                                 const double *ADp, const double *b,
                                 unsigned long long *inf, int64_t vs,
                                 uint32_t vact) {
  grid_wait();
  if (batch_skip(vact)) return;
  x += blockIdx.y * vs;
  b += blockIdx.y * vs;
  inf += 8 * blockIdx.y;
  const int64_t gid  = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t row  = gid / G;
  const int     lane = threadIdx.x % G;
  const bool    act  = row < n;
  double        s = 0.0, a = 0.0;
  if (act)
    for (int64_t e = Kp[row] + lane; e < Kp[row + 1]; e += G) {
      const int32_t j = Kj[e];
      s += Korig[e] * (x[j] * ADp[j]);
      a += fabs(Korig[e]);
    }
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) {
    s += __shfl_xor_sync(0xffffffffu, s, o, G);
    a += __shfl_xor_sync(0xffffffffu, a, o, G);
  }
  const bool lead = act && lane == 0;
  warp_max_abs(inf + 0, lead ? b[row] - s : 0.0, lead);
  warp_max_abs(inf + 1, lead ? a : 0.0, lead);
  warp_max_abs(inf + 2, lead ? x[row] * ADp[row] : 0.0, lead);
  warp_max_abs(inf + 3, lead ? b[row] : 0.0, lead);
}

// y = a * x.
__global__ void k_scale(int64_t n, const double *x, double a, double *y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] = x[i] * a;
}

// d *= scale; inf[0] = max|d|; inf[1] = max|x_old|; x += d
// (gmres_ir.hpp:574-577).
__global__ void k_ir_update(int64_t n, double *d, double scale, double *x,
                            const double *w, unsigned long long *inf) {
  const int64_t i   = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool    act = i < n;
  double        di = 0.0, xi = 0.0, wi = 1.0;
  if (act) {
    di   = d[i] * scale;
    xi   = x[i];
    d[i] = di;
    x[i] = xi + di;
    if (w) wi = w[i];
  }
  warp_max_abs(inf + 0, di * wi, act);
  warp_max_abs(inf + 1, xi * wi, act);
}

// x <- x rounded to float32 (1), bfloat16 (2) or float16 (3).
__global__ void k_round_to(int64_t n, int prec, double *x) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double v = x[i];
  if (prec == 1)
    x[i] = static_cast<double>(__double2float_rn(v));
  else if (prec == 2)
    x[i] = static_cast<double>(__bfloat162float(__double2bfloat16(v)));
  else if (prec == 3)
    x[i] = static_cast<double>(__half2float(__double2half(v)));
}

// bs[i] = b[perm[i]] * AD[perm[i]]; ADp[i] = AD[perm[i]]; bp[i] = b[perm[i]];
// inf[0] = max|bs|.
// Batched: b, bs, bp of vector k at k*vs; ADp is written by k == 0 only.
__global__ void k_rhs_in(int64_t n, const int64_t *perm, const double *AD,
                         const double *b, double *bs, double *ADp, double *bp,
                         unsigned long long *inf, int64_t vs) {
  grid_wait();
  b += blockIdx.y * vs;
  bs += blockIdx.y * vs;
  bp += blockIdx.y * vs;
  inf += 8 * blockIdx.y;
  if (blockIdx.y != 0) ADp = nullptr;
  const int64_t i   = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const bool    act = i < n;
  double        v   = 0.0;
  if (act) {
    const int64_t o = perm[i];
    const double  a = AD[o];
    v               = b[o] * a;
    bs[i]           = v;
    if (ADp) ADp[i] = a;
    bp[i]           = b[o];
  }
  warp_max_abs(inf, v, act);
}

// out[perm[i]] = x[i] * ADp[i] (ADp NULL: out[perm[i]] = x[i]).
__global__ void k_sol_out(int64_t n, const int64_t *perm, const double *ADp,
                          const double *x, double *out, int64_t vs) {
  grid_wait();
  x += blockIdx.y * vs;
  out += blockIdx.y * vs;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) out[perm[i]] = ADp ? x[i] * ADp[i] : x[i];
}

// ---------------------------------------------------------------------------
// Host wrappers.
static unsigned blocks_for(int64_t n, int t) {
  return static_cast<unsigned>(std::max<int64_t>(1, (n + t - 1) / t));
}

void VecOps::allocate(int64_t n_, int batch_) {
  n     = n_;
  batch = std::max(batch_, 1);
  infbits.resize(sizeof(unsigned long long) * 8 * batch);
}

// Zeroes slots [first, first + cnt) of banks 0 .. nb-1.
static void clear_slots(unsigned long long *bits, int nb, int first, int cnt, cudaStream_t s) {
  if (nb == 1)
    MPIR_CUDA(cudaMemsetAsync(bits + first, 0, cnt * sizeof(unsigned long long), s));
  else
    MPIR_CUDA(cudaMemset2DAsync(bits + first, 8 * sizeof(unsigned long long), 0,
                                cnt * sizeof(unsigned long long), nb, s));
}

static dim3 grid_b(int64_t work, int threads, int nb) {
  return dim3(blocks_for(work, threads), static_cast<unsigned>(nb), 1);
}

constexpr uint32_t kAll = 0xffffffffu;

void VecOps::spmv(int nb, const int64_t *Kp, const int32_t *Kj, const double *Kv, const double *x,
                  double *y, cudaStream_t s) {
  constexpr int G = 8;
  launch_chained(n, k_spmv<G, 0>, 1, grid_b(n * G, 256, nb), 256, 0, s, n, Kp, Kj, Kv, x, nullptr, y, nullptr, n,
                 kAll);
}

void VecOps::residual(int nb, uint32_t act, const int64_t *Kp, const int32_t *Kj, const double *Kv,
                      const double *x, const double *b, double *r, bool dd, bool clear, cudaStream_t s) {
  constexpr int       G   = 8;
  unsigned long long *inf = infbits.as<unsigned long long>();
  if (clear) clear_slots(inf, nb, 0, 1, s);
  launch_chained(n, dd ? k_spmv<G, 2> : k_spmv<G, 1>, 1, grid_b(n * G, 256, nb), 256, 0, s, n, Kp, Kj, Kv, x, b,
                 r, inf, n, act);
}

void VecOps::backward_terms(int nb, const int64_t *Kp, const int32_t *Kj, const double *Korig,
                            const double *x, const double *ADp, const double *bp, cudaStream_t s) {
  constexpr int       G   = 8;
  unsigned long long *inf = infbits.as<unsigned long long>();
  clear_slots(inf, nb, 4, 4, s);
  launch_chained(n, k_backward_terms<G>, 1, grid_b(n * G, 256, nb), 256, 0, s, n, Kp, Kj, Korig, x, ADp, bp, inf + 4, n,
         kAll);
}

void VecOps::scale(const double *x, double a, double *y, cudaStream_t s) {
  launch(k_scale, blocks_for(n, 256), 256, 0, s, n, x, a, y);
}

void VecOps::ir_update(double *d, double scale, double *x, cudaStream_t s, const double *w) {
  unsigned long long *inf = infbits.as<unsigned long long>() + 1;
  MPIR_CUDA(cudaMemsetAsync(inf, 0, 2 * sizeof(unsigned long long), s));
  launch(k_ir_update, blocks_for(n, 256), 256, 0, s, n, d, scale, x, w, inf);
}

void VecOps::round_to(int prec, double *x, cudaStream_t s) {
  if (prec < 1 || prec > 3) return;
  launch(k_round_to, blocks_for(n, 256), 256, 0, s, n, prec, x);
}

void VecOps::rhs_in(int nb, const int64_t *perm, const double *AD, const double *b, double *bs,
                    double *ADp, double *bp, cudaStream_t s) {
  unsigned long long *inf = infbits.as<unsigned long long>();
  clear_slots(inf, nb, 3, 1, s);
  launch_chained(n, k_rhs_in, 1, grid_b(n, 256, nb), 256, 0, s, n, perm, AD, b, bs, ADp, bp, inf + 3, n);
}

void VecOps::sol_out(int nb, const int64_t *perm, const double *ADp, const double *x, double *out,
                     cudaStream_t s) {
  launch_chained(n, k_sol_out, 1, grid_b(n, 256, nb), 256, 0, s, n, perm, ADp, x, out, n);
}

void VecOps::read_inf(int nb, double *h, cudaStream_t s) {
  static_assert(sizeof(double) == sizeof(unsigned long long), "bit copy");
  MPIR_CUDA(cudaMemcpyAsync(h, infbits.as<void>(), nb * 8 * sizeof(double), cudaMemcpyDeviceToHost, s));
  MPIR_CUDA(cudaStreamSynchronize(s));
}

}  // namespace mpir
