// PrecondGmres (gmres_ir.hpp:636-741) on the device: the modified Gram-Schmidt
// step, the Givens rotations and the stop tests, one launch per inner step.
//
// A step's k + 2 reductions depend on one another, and at these sizes each is
// latency, not bandwidth: as separate launches (one per reduction, a copy of
// the column to the host and a synchronisation for its rotations) a step of
// k = 4 took about 40 us beside the preconditioner.  Here one thread-block
// cluster per vector keeps w in registers and runs the whole step: a reduction
// is a block reduction, one exchange through distributed shared memory and one
// cluster barrier (about 1 us).  Systems of up to 8,192 unknowns take one CTA,
// which needs neither; a cluster of 8 (16 from 65,536 on) covers the rest, with
// the entries beyond its registers (512 threads x 16 a CTA) in global memory.
// One thread applies the rotations and decides whether to go on; these kernels
// and the solves of a step that is not taken return at once, so the host may
// queue the next step before it knows (that step's SpMV does run, once an inner
// loop: 8.5 us at n = 40,960).
//
// Measured outside the triangular solves: n = 1,280, 5 inner steps in two inner
// loops, 0.46 ms a solve as separate launches, 0.15 here; n = 40,960 (8 CTAs), 7
// steps in three, 0.9 -> 0.4 ms; three vectors of n = 40,951, 9 steps in three,
// 1.3 -> 0.5 ms.
//
// A cluster's 16 SMs read the basis at about 1.3 TB/s.  Up to four vectors of more
// than 200,000 entries are therefore swept by the whole chip, one launch a basis
// vector (k_wide_*), whose partial sums the next one adds up; the cluster keeps the
// norms' slow cases, the second sweep and the rotations.  80 steps over up to 40
// basis vectors, solves included, as separate reductions and updates, by a cluster
// alone, so (ms): n = 200,000 32.6, 28.5, -; 327,680 44.8, 51.8, 39.3; 500,000 64.6, 82.3,
// 56.8; 4 million 490, 784, 423.
//
// Sums run in a fixed order (threads, warps, CTAs), so results are
// reproducible.  Norms are sqrt of the sum of squares, or, where that sum is
// not well inside the range of float64, the scaled form of Dnrm2
// (ops.hpp:231-264).
#include <cmath>

#include "arnoldi.hpp"
#include "common.cuh"

namespace mpir {

namespace {

constexpr int kThreads = 512;
constexpr int kRegs    = 16;  // entries of w a thread keeps
constexpr int kWarps   = kThreads / 32;

struct ArnoldiArgs {
  int64_t    n, m, cap, vs, block, stride;  // steps allowed, laid out
  double    *V, *state;
  double     tol;
  GmresMail *mail;
  double    *wide;  // kWideStride a vector: WideScratch, partial sums (NULL: no chip-wide kernels)
};

// Vectors of more than kWideFrom entries, up to kWideVectors of them, are swept by
// the whole chip (k_wide_*), one launch a basis vector, the others by a cluster each.
constexpr int64_t kWideFrom    = 200000;
constexpr int     kWideVectors = 4;
constexpr int     kWideCtas    = 148;
constexpr int     kWideStride  = 4 + 4 * kWideCtas;
struct WideScratch {
  double  ss;   // |w|^2 before the sweep
  double  f;    // factor of k_wide_scale
  int32_t odd;  // |w|^2 has left the range in which it is accurate: the step is the cluster's
  int32_t pad[3];
};
static_assert(sizeof(WideScratch) == 32, "four doubles");

struct StateView {
  GmresCtl *ctl;
  double   *R, *c, *s, *g, *y, *col;
  __host__ __device__ StateView(double *p, int64_t cap) {
    ctl = reinterpret_cast<GmresCtl *>(p);
    R   = p + 4;
    c   = R + cap * (cap + 1) / 2;
    s   = c + cap;
    g   = s + cap;
    y   = g + cap + 1;
    col = y + cap;
  }
  __device__ StateView(const ArnoldiArgs &a, int vec) : StateView(a.state + vec * a.stride, a.cap) {}
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
// (Not the .aligned forms: a warp's lanes may come here from a loop that they
// left at different turns.)
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// A CTA's shared memory exists for the others of its cluster only once it is
// known to have started: arrive at the start, wait before the first
// cluster_put (the vectors' first loads lie in between).  Nothing is handed
// over, so the arrival orders no memory.
__device__ __forceinline__ void cluster_arrive() {
  if (cluster_size() > 1) asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
  if (cluster_size() > 1) asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}
// One double into CTA `rank`'s copy of a shared variable.
__device__ __forceinline__ void cluster_put(double *p, uint32_t rank, double v) {
  uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(p)), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(v) : "memory");
}

struct RedShared {
  double warp[2][kWarps];
  double slot[2][16][2];  // by the parity of the reduction, by CTA
};

// Sums (or, MAX, maxima) of a and b over the cluster, in every thread.
template <bool MAX>
struct Reducer {
  RedShared &S;
  int       &turn;
  __device__ __forceinline__ static double op(double x, double y) { return MAX ? (x > y ? x : y) : x + y; }
  __device__ __forceinline__ void run(double &a, double &b) {
    const unsigned full = 0xffffffffu;
    const int      warp = threadIdx.x / 32, lane = threadIdx.x % 32, C = cluster_size();
    const int      t = turn & 1;
    turn++;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a = op(a, __shfl_xor_sync(full, a, o));
      b = op(b, __shfl_xor_sync(full, b, o));
    }
    if (lane == 0) {
      S.warp[0][warp] = a;
      S.warp[1][warp] = b;
    }
    __syncthreads();
    if (warp == 0) {
      a = S.warp[0][lane % kWarps];
      b = S.warp[1][lane % kWarps];
#pragma unroll
      for (int o = kWarps / 2; o > 0; o >>= 1) {
        a = op(a, __shfl_xor_sync(full, a, o));
        b = op(b, __shfl_xor_sync(full, b, o));
      }
      if (C == 1) {
        if (lane == 0) {
          S.slot[t][0][0] = a;
          S.slot[t][0][1] = b;
        }
      } else if (lane < C) {
        cluster_put(&S.slot[t][cluster_rank()][0], lane, a);
        cluster_put(&S.slot[t][cluster_rank()][1], lane, b);
      }
    }
    if (C == 1)
      __syncthreads();
    else
      cluster_sync();
    a = S.slot[t][0][0];
    b = S.slot[t][0][1];
    for (int r = 1; r < C; r++) {
      a = op(a, S.slot[t][r][0]);
      b = op(b, S.slot[t][r][1]);
    }
  }
};

// A vector spread over the cluster: entry j of a thread is (j C + rank) 512 +
// tid; the first kRegs in registers, the rest in global memory.
struct Spread {
  int64_t n, i0, step;
  __device__ Spread(int64_t n_) : n(n_) {
    step = static_cast<int64_t>(cluster_size()) * kThreads;
    i0   = static_cast<int64_t>(cluster_rank()) * kThreads + threadIdx.x;
  }
  __device__ __forceinline__ void load(double (&w)[kRegs], const double *p) const {
#pragma unroll
    for (int j = 0; j < kRegs; j++) w[j] = i0 + j * step < n ? p[i0 + j * step] : 0.0;
  }
  // f(i) for the entries beyond the registers.
  template <class F>
  __device__ __forceinline__ void rest(F f) const {
#pragma unroll 4
    for (int64_t i = i0 + kRegs * step; i < n; i += step) f(i);
  }
  template <class F>
  __device__ __forceinline__ void regs(F f) const {
#pragma unroll
    for (int j = 0; j < kRegs; j++)
      if (i0 + j * step < n) f(j, i0 + j * step);
  }
};

// sqrt(ss), ss the sum of squares of w, or the scaled norm where ss has left
// the range in which that is accurate.
__device__ double safe_norm(double ss, const Spread &sp, const double (&w)[kRegs], const double *wg,
                            RedShared &S, int &turn) {
  if (ss > 1e-280 && ss < 1e280) return sqrt(ss);
  if (!(ss == ss)) return ss;
  double mx = 0.0, none = 0.0;
#pragma unroll
  for (int j = 0; j < kRegs; j++) mx = fmax(mx, fabs(w[j]));
  sp.rest([&](int64_t i) { mx = fmax(mx, fabs(wg[i])); });
  Reducer<true>{S, turn}.run(mx, none);
  if (mx == 0.0 || !isfinite(mx)) return mx;
  double q = 0.0;
  none     = 0.0;
#pragma unroll
  for (int j = 0; j < kRegs; j++) q += (w[j] / mx) * (w[j] / mx);
  sp.rest([&](int64_t i) { q += (wg[i] / mx) * (wg[i] / mx); });
  Reducer<false>{S, turn}.run(q, none);
  return mx * sqrt(q);
}

// x = d, or x += d f with the largest |d f| and |x before| (gmres_ir.hpp:574-577).  NaN
// counts as above infinity, as in the max-norms of the vector kernels.
__device__ __forceinline__ void refine(double d, double f, int update, double &x, double &dm, double &xm) {
  if (!update) {
    x = d;
    return;
  }
  const double di = d * f, xi = x;
  dm = fabs(di) > dm || !(di == di) ? fabs(di) : dm;
  xm = fabs(xi) > xm || !(xi == xi) ? fabs(xi) : xm;
  x  = xi + di;
}

__device__ __forceinline__ WideScratch *wide_scratch(const ArnoldiArgs &a, int vec) {
  return reinterpret_cast<WideScratch *>(a.wide + static_cast<int64_t>(kWideStride) * vec);
}
// The CTAs' partial sums `which` of launches of parity t; added in a fixed order, in
// every thread.
__device__ __forceinline__ double *wide_part(const ArnoldiArgs &a, int vec, int t, int which) {
  return a.wide + static_cast<int64_t>(kWideStride) * vec + 4 + (2 * t + which) * kWideCtas;
}
__device__ __forceinline__ double wide_sum(const double *p) {
  __shared__ double out;
  if (threadIdx.x < 32) {
    double s = 0.0;
#pragma unroll
    for (int q = 0; q < (kWideCtas + 31) / 32; q++) {
      const int i = threadIdx.x + 32 * q;
      s += i < kWideCtas ? __ldcg(p + i) : 0.0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) out = s;
  }
  __syncthreads();
  const double s = out;
  __syncthreads();
  return s;
}
// The CTA's sum of v into its place.
__device__ __forceinline__ void wide_store(double *p, double v) {
  __shared__ double warp[kWarps];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (threadIdx.x % 32 == 0) warp[threadIdx.x / 32] = v;
  __syncthreads();
  if (threadIdx.x < 32) {
    v = threadIdx.x < kWarps ? warp[threadIdx.x] : 0.0;
#pragma unroll
    for (int o = kWarps / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (threadIdx.x == 0) p[blockIdx.x] = v;
  }
  __syncthreads();
}
// f(i) for the entries of one CTA of the chip.
template <class F>
__device__ __forceinline__ void wide_each(int64_t n, F f) {
  constexpr int64_t step = static_cast<int64_t>(kWideCtas) * kThreads;
#pragma unroll 4
  for (int64_t i = blockIdx.x * static_cast<int64_t>(kThreads) + threadIdx.x; i < n; i += step) f(i);
}

// V_0 = b fac with |V_0|^2 (begin), or |V_0|^2 of what is there.
__global__ void __launch_bounds__(kThreads)
    k_wide_norm(const ArnoldiArgs a, uint32_t act, const double *b, const VecFactors fac) {
  grid_wait();
  const int vec = blockIdx.y;
  if (b ? !(act >> vec & 1u) : StateView(a, vec).ctl->active == 0) return;
  const double f  = fac.v[vec];
  double      *w0 = a.V + vec * a.vs, ss = 0.0;
  wide_each(a.n, [&](int64_t i) {
    double x = w0[i];
    if (b) {
      x     = b[vec * a.vs + i] * f;
      w0[i] = x;
    }
    ss += x * x;
  });
  wide_store(wide_part(a, vec, 0, 1), ss);
}

// Launch j = 0 .. k + 1 of step k: h_{j-1} from the launch before, w -= h_{j-1}
// v_{j-1}, the partial sums of w v_j, in the last one of |w|^2 (in the first also).
__global__ void __launch_bounds__(kThreads) k_wide_sweep(const ArnoldiArgs a, int64_t k, int64_t j) {
  grid_wait();
  const int    vec = blockIdx.y, t = j & 1;
  StateView    st(a, vec);
  WideScratch *sc = wide_scratch(a, vec);
  if (st.ctl->active == 0 || (j > 1 && sc->odd)) return;
  const bool lead = blockIdx.x == 0 && threadIdx.x == 0;
  double     h = 0.0, s = 0.0, ss = 0.0;
  if (j > 0) {
    h = wide_sum(wide_part(a, vec, 1 - t, 0));
    if (j == 1) {
      ss             = wide_sum(wide_part(a, vec, 0, 1));
      const bool odd = !(ss > 1e-280 && ss < 1e280);
      if (lead) {
        sc->ss  = ss;
        sc->odd = odd;
      }
      if (odd) return;
      ss = 0.0;
    }
    if (lead) st.col[j - 1] = h;
  }
  double       *V = a.V + vec * a.vs, *w = V + (k + 1) * a.block;
  const double *vb = V + (j - 1) * a.block, *vj = V + j * a.block;
  if (j == 0) {
    wide_each(a.n, [&](int64_t i) {
      const double x = w[i];
      s += x * vj[i];
      ss += x * x;
    });
    wide_store(wide_part(a, vec, 0, 1), ss);
  } else if (j <= k) {
    wide_each(a.n, [&](int64_t i) {
      const double x = w[i] - vb[i] * h;
      w[i]           = x;
      s += x * vj[i];
    });
  } else {
    wide_each(a.n, [&](int64_t i) {
      const double x = w[i] - vb[i] * h;
      w[i]           = x;
      s += x * x;
    });
  }
  wide_store(wide_part(a, vec, t, 0), s);
}

// V_j *= the factor that the step (or first) left.
__global__ void __launch_bounds__(kThreads) k_wide_scale(const ArnoldiArgs a, int64_t j) {
  grid_wait();
  const int vec = blockIdx.y;
  if (StateView(a, vec).ctl->active == 0) return;
  const double f = wide_scratch(a, vec)->f;
  double      *w = a.V + vec * a.vs + j * a.block;
  wide_each(a.n, [&](int64_t i) { w[i] *= f; });
}

// The combination of the basis (k_gmres_end).
__global__ void __launch_bounds__(kThreads)
    k_wide_end(const ArnoldiArgs a, uint32_t act, double *x, int update, const VecFactors fac,
               unsigned long long *inf) {
  grid_wait();
  const int vec = blockIdx.y;
  if (!(act >> vec & 1u)) return;
  const StateView st(a, vec);
  const int64_t   k  = st.ctl->k;
  const double    f  = fac.v[vec];
  const double   *V  = a.V + vec * a.vs;
  double         *xv = x + vec * a.vs, dm = 0.0, xm = 0.0;
  wide_each(a.n, [&](int64_t i) {
    double d = 0.0;
#pragma unroll 4
    for (int64_t j = 0; j < k; j++) d += V[j * a.block + i] * st.y[j];
    refine(d, f, update, xv[i], dm, xm);
  });
  if (!update) return;
  unsigned long long b0 = __double_as_longlong(dm), b1 = __double_as_longlong(xm);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long c0 = __shfl_xor_sync(0xffffffffu, b0, o), c1 = __shfl_xor_sync(0xffffffffu, b1, o);
    b0 = c0 > b0 ? c0 : b0;
    b1 = c1 > b1 ? c1 : b1;
  }
  if (threadIdx.x % 32 == 0) {
    atomicMax(inf + 8 * vec + 1, b0);
    atomicMax(inf + 8 * vec + 2, b1);
  }
}

// A CTA of a cluster must not exit while another may still write to its shared
// memory or wait for it.
__device__ __forceinline__ void leave() {
  if (cluster_size() > 1) cluster_sync();
}

template <bool WIDE>
__global__ void __launch_bounds__(kThreads)
    k_gmres_begin(const ArnoldiArgs a, uint32_t act, const double *b, const VecFactors fac) {
  grid_wait();
  __shared__ RedShared S;
  int                  turn = 0;
  const int            vec  = blockIdx.y;
  StateView            st(a, vec);
  const bool           lead = cluster_rank() == 0 && threadIdx.x == 0;
  if (!(act >> vec & 1u)) {
    if (lead) {
      *st.ctl               = GmresCtl{0.0, 0, 0, 0, 0, {0, 0}};
      a.mail->active[0][vec] = a.mail->active[1][vec] = 0;
    }
    return;
  }
  cluster_arrive();
  const Spread  sp(a.n);
  const double  f  = fac.v[vec];
  const double *bv = b + vec * a.vs;
  double       *w0 = a.V + vec * a.vs, w[kRegs], ss = 0.0, none = 0.0;
  if (WIDE) {
    sp.load(w, w0);
    ss = wide_sum(wide_part(a, vec, 0, 1));
    cluster_wait();
  } else {
    sp.load(w, bv);
#pragma unroll
    for (int j = 0; j < kRegs; j++) {
      w[j] *= f;
      ss += w[j] * w[j];
    }
    sp.regs([&](int j, int64_t i) { w0[i] = w[j]; });
    sp.rest([&](int64_t i) {
      const double x = bv[i] * f;
      w0[i]          = x;
      ss += x * x;
    });
    cluster_wait();
    Reducer<false>{S, turn}.run(ss, none);
  }
  const double rho = safe_norm(ss, sp, w, w0, S, turn);
  if (lead) {
    const int32_t go       = !(rho < a.tol);  // gmres_ir.hpp:655-657
    *st.ctl                = GmresCtl{rho, 0, go, 0, go, {0, 0}};
    a.mail->active[0][vec] = a.mail->active[1][vec] = go;
  }
  leave();
}

template <bool WIDE>
__global__ void __launch_bounds__(kThreads) k_gmres_first(const ArnoldiArgs a) {
  grid_wait();
  __shared__ RedShared S;
  int                  turn = 0;
  const int            vec  = blockIdx.y;
  StateView            st(a, vec);
  if (st.ctl->active == 0) return;
  cluster_arrive();
  const Spread sp(a.n);
  double      *w0 = a.V + vec * a.vs, w[kRegs], ss = 0.0, none = 0.0;
  sp.load(w, w0);
  if (WIDE) {
    ss = wide_sum(wide_part(a, vec, 0, 1));
    cluster_wait();
  } else {
#pragma unroll
    for (int j = 0; j < kRegs; j++) ss += w[j] * w[j];
    sp.rest([&](int64_t i) { ss += w0[i] * w0[i]; });
    cluster_wait();
    Reducer<false>{S, turn}.run(ss, none);
  }
  const double rho = safe_norm(ss, sp, w, w0, S, turn), f = 1 / rho;
  if (WIDE) {
    if (cluster_rank() == 0 && threadIdx.x == 0) wide_scratch(a, vec)->f = f;
  } else {
    sp.regs([&](int j, int64_t i) { w0[i] = w[j] * f; });
    sp.rest([&](int64_t i) { w0[i] *= f; });
  }
  leave();  // every CTA has read the active flag
  if (cluster_rank() == 0 && threadIdx.x == 0) {
    st.g[0]         = rho;
    st.ctl->rho     = rho;
    st.ctl->active  = a.m > 0 && rho > a.tol;
  }
}

// One inner step (gmres_ir.hpp:664-726): |w|, then for each basis vector v_j
// h = w v_j and w -= h v_j, each pass summing for the next one (the loads of
// v_{j+1} before its reduction); a second sweep where Brown and Hindmarsh's test
// asks for it; w /= |w|; the rotations.
template <bool WIDE>
__global__ void __launch_bounds__(kThreads) k_gmres_step(const ArnoldiArgs a, int64_t k) {
  grid_wait();
  __shared__ RedShared S;
  int                  turn = 0;
  const int            vec  = blockIdx.y, lane = threadIdx.x % 32;
  StateView            st(a, vec);
  const bool           lead = cluster_rank() == 0 && threadIdx.x == 0;
  if (st.ctl->active == 0) {
    if (lead) a.mail->active[k & 1][vec] = 0;
    return;
  }
  cluster_arrive();
  const Spread sp(a.n);
  double      *V = a.V + vec * a.vs, *wg = V + (k + 1) * a.block;
  double       w[kRegs], v[kRegs];
  const bool   swept = WIDE && !wide_scratch(a, vec)->odd;  // pass 0 is done
  sp.load(w, wg);
  double ss = 0.0, h = 0.0;
  if (swept) {
    ss = wide_scratch(a, vec)->ss;
    h  = wide_sum(wide_part(a, vec, (k + 1) & 1, 0));
    cluster_wait();
  } else {
    sp.load(v, V);
#pragma unroll
    for (int j = 0; j < kRegs; j++) {
      ss += w[j] * w[j];
      h += w[j] * v[j];
    }
    sp.rest([&](int64_t i) {
      ss += wg[i] * wg[i];
      h += wg[i] * V[i];
    });
    cluster_wait();
    Reducer<false>{S, turn}.run(ss, h);
  }
  // (Of a swept w, which is not what ss was summed of, ss is within the range.)
  const double normav = safe_norm(ss, sp, w, wg, S, turn);
  double       normw  = 0.0;
  int32_t      reorth = 0;
  for (int pass = 0;; pass++) {
    for (int64_t j = swept && pass == 0 ? k + 1 : 0; j <= k; j++) {
      if (lead) st.col[j] = pass == 0 ? h : st.col[j] + h;
      const double *vj = V + j * a.block, *vn = vj + a.block;
      const double  hj = h;
      const bool    more = j < k;
#pragma unroll
      for (int q = 0; q < kRegs; q++) w[q] -= v[q] * hj;
      if (more) sp.load(v, vn);
      double t = 0.0, none = 0.0;
#pragma unroll
      for (int q = 0; q < kRegs; q++) t += w[q] * (more ? v[q] : w[q]);
      sp.rest([&](int64_t i) {
        const double x = wg[i] - vj[i] * hj;
        wg[i]          = x;
        t += x * (more ? vn[i] : x);
      });
      Reducer<false>{S, turn}.run(t, none);
      h = t;
    }
    normw = safe_norm(h, sp, w, wg, S, turn);
    // Brown/Hindmarsh, gmres_ir.hpp:683
    if (pass > 0 || !(normav + 0.001 * normw == normav)) break;
    reorth = 1;
    sp.load(v, V);
    double t = 0.0, none = 0.0;
#pragma unroll
    for (int q = 0; q < kRegs; q++) t += w[q] * v[q];
    sp.rest([&](int64_t i) { t += wg[i] * V[i]; });
    Reducer<false>{S, turn}.run(t, none);
    h = t;
  }
  const double f = normw != 0 ? 1 / normw : 1.0;
  if (WIDE) {  // scaled by k_wide_scale, where the loop goes on
    if (lead) wide_scratch(a, vec)->f = f;
    if (!swept || reorth) sp.regs([&](int j, int64_t i) { wg[i] = w[j]; });
  } else {
    sp.regs([&](int j, int64_t i) { wg[i] = w[j] * f; });
    sp.rest([&](int64_t i) { wg[i] *= f; });
  }
  leave();  // every CTA has read the active flag
  if (cluster_rank() != 0 || threadIdx.x >= 32) return;
  // The column's rotations, by one warp: 32 of them are loaded at a time, the
  // chain over them runs in registers.
  __syncwarp();
  double       *R = st.R + k * (k + 1) / 2;
  double        hj = __shfl_sync(0xffffffffu, lane == 0 ? st.col[0] : 0.0, 0);  // h(j, k) so far
  for (int64_t j0 = 0; j0 < k; j0 += 32) {
    const bool   ok = j0 + lane < k;
    const double cj = ok ? st.c[j0 + lane] : 0.0, sj = ok ? st.s[j0 + lane] : 0.0;
    const double hn = ok ? __ldcg(st.col + j0 + lane + 1) : 0.0;
    double       out = 0.0;
    const int    cnt = static_cast<int>(k - j0 < 32 ? k - j0 : 32);
    for (int q = 0; q < cnt; q++) {
      const double c1 = __shfl_sync(0xffffffffu, cj, q), s1 = __shfl_sync(0xffffffffu, sj, q);
      const double h1 = __shfl_sync(0xffffffffu, hn, q);
      const double w1 = c1 * hj - s1 * h1, w2 = s1 * hj + c1 * h1;
      if (lane == q) out = w1;
      hj = w2;
    }
    if (ok) R[j0 + lane] = out;
  }
  if (lane != 0) return;
  // Dnrm2 of {h_kk, h_k+1,k}, walked last to first as ops.hpp:243 does.
  double       scale = 0.0, ssq = 1.0;
  const double pr[2] = {hj, normw};
#pragma unroll
  for (int q = 1; q >= 0; q--)
    if (pr[q] != 0.0) {
      const double x = fabs(pr[q]);
      if (scale < x) {
        ssq   = 1.0 + ssq * ((scale / x) * (scale / x));
        scale = x;
      } else {
        ssq = ssq + ((x / scale) * (x / scale));
      }
    }
  const double nu = scale * sqrt(ssq);
  double       gk = st.g[k], gn = 0.0;
  if (nu != 0) {
    const double c = hj / nu, s = -normw / nu;
    st.c[k] = c;
    st.s[k] = s;
    hj      = c * hj - s * normw;
    gn      = s * gk;
    gk      = c * gk;
  } else {
    st.c[k] = 0.0;
    st.s[k] = 0.0;
  }
  R[k]           = hj;
  st.g[k]        = gk;
  st.g[k + 1]    = gn;
  const double r = fabs(gn);
  const int32_t go = k + 1 < a.m && r > a.tol;
  st.ctl->rho    = r;
  st.ctl->k      = static_cast<int32_t>(k + 1);
  st.ctl->active = go;
  st.ctl->reorth += reorth;
  a.mail->active[k & 1][vec] = go;
}

template <bool WIDE>
__global__ void __launch_bounds__(kThreads)
    k_gmres_end(const ArnoldiArgs a, uint32_t act, double *x, int update, const VecFactors fac,
                unsigned long long *inf) {
  grid_wait();
  __shared__ RedShared S;
  const int            vec = blockIdx.y, tid = threadIdx.x;
  if (!(act >> vec & 1u)) return;
  StateView     st(a, vec);
  const int64_t k = st.ctl->k;
  // y = R^{-1} g by columns, in the leading CTA.
  if (cluster_rank() == 0) {
    for (int64_t j = tid; j < k; j += kThreads) st.y[j] = st.g[j];
    __syncthreads();
    for (int64_t i = k - 1; i >= 0; i--) {
      const double *R  = st.R + i * (i + 1) / 2;
      const double  yi = st.y[i] / R[i];
      __syncthreads();
      for (int64_t j = tid; j <= i; j += kThreads) st.y[j] = j == i ? yi : st.y[j] - R[j] * yi;
      __syncthreads();
    }
    if (tid == 0) {
      a.mail->k[vec]      = static_cast<int32_t>(k);
      a.mail->reorth[vec] = st.ctl->reorth;
      a.mail->began[vec]  = st.ctl->began;
    }
  }
  if (WIDE) {  // the rest is k_wide_end's
    if (update && cluster_rank() == 0 && tid < 3) inf[8 * vec + tid] = 0;
    return;
  }
  if (cluster_size() > 1)
    cluster_sync();
  else
    __syncthreads();
  const Spread  sp(a.n);
  const double  f  = fac.v[vec];
  const double *V  = a.V + vec * a.vs;
  double       *xv = x + vec * a.vs, d[kRegs], dm = 0.0, xm = 0.0;
#pragma unroll
  for (int j = 0; j < kRegs; j++) d[j] = 0.0;
  // (y is written by another CTA: not through the read-only path.)
  for (int64_t j = 0; j < k; j++) {
    const double  yj = __ldcg(st.y + j);
    const double *vj = V + j * a.block;
    sp.regs([&](int q, int64_t i) { d[q] += vj[i] * yj; });
  }
  auto put = [&](double dv, int64_t i) { refine(dv, f, update, xv[i], dm, xm); };
  sp.regs([&](int q, int64_t i) { put(d[q], i); });
  sp.rest([&](int64_t i) {
    double dv = 0.0;
    for (int64_t j = 0; j < k; j++) dv += V[j * a.block + i] * __ldcg(st.y + j);
    put(dv, i);
  });
  if (!update) return;
  // max over the cluster on the bit patterns (the order of non-negative
  // doubles, NaN above all)
  {
    const unsigned      full = 0xffffffffu;
    unsigned long long  b0 = __double_as_longlong(dm), b1 = __double_as_longlong(xm);
    __shared__ unsigned long long sb[2][kWarps];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long c0 = __shfl_xor_sync(full, b0, o), c1 = __shfl_xor_sync(full, b1, o);
      b0 = c0 > b0 ? c0 : b0;
      b1 = c1 > b1 ? c1 : b1;
    }
    if (tid % 32 == 0) {
      sb[0][tid / 32] = b0;
      sb[1][tid / 32] = b1;
    }
    __syncthreads();
    if (tid == 0) {
      for (int q = 1; q < kWarps; q++) {
        b0 = sb[0][q] > b0 ? sb[0][q] : b0;
        b1 = sb[1][q] > b1 ? sb[1][q] : b1;
      }
      if (cluster_size() > 1) {
        cluster_put(&S.slot[0][cluster_rank()][0], 0, __longlong_as_double(static_cast<long long>(b0)));
        cluster_put(&S.slot[0][cluster_rank()][1], 0, __longlong_as_double(static_cast<long long>(b1)));
      }
    }
    if (cluster_size() > 1) cluster_sync();
    if (cluster_rank() == 0 && tid == 0) {
      if (cluster_size() > 1) {
        b0 = b1 = 0;
        for (uint32_t r = 0; r < cluster_size(); r++) {
          const unsigned long long c0 = __double_as_longlong(S.slot[0][r][0]),
                                   c1 = __double_as_longlong(S.slot[0][r][1]);
          b0 = c0 > b0 ? c0 : b0;
          b1 = c1 > b1 ? c1 : b1;
        }
      }
      inf[8 * vec]     = 0;
      inf[8 * vec + 1] = b0;
      inf[8 * vec + 2] = b1;
    }
  }
}

ArnoldiArgs make_args(int64_t n, int64_t m, int64_t cap, int64_t stride, double *V, int64_t block, double *state,
                      double tol, GmresMail *mail, double *wide) {
  return ArnoldiArgs{n, m, cap, n, block, stride, V, state, tol, mail, wide};
}

// Clusters of more than 8 CTAs have to be allowed, on each device.
void allow_large_clusters() {
  for (auto *f :
       {reinterpret_cast<const void *>(k_gmres_begin<false>), reinterpret_cast<const void *>(k_gmres_first<false>),
        reinterpret_cast<const void *>(k_gmres_step<false>), reinterpret_cast<const void *>(k_gmres_end<false>),
        reinterpret_cast<const void *>(k_gmres_begin<true>), reinterpret_cast<const void *>(k_gmres_first<true>),
        reinterpret_cast<const void *>(k_gmres_step<true>), reinterpret_cast<const void *>(k_gmres_end<true>)})
    MPIR_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
}

}  // namespace

Arnoldi::~Arnoldi() {
  if (mail_) pinned_free(mail_, sizeof(GmresMail));
}

void Arnoldi::allocate(int64_t n, int64_t m, int vectors) {
  n_       = n;
  m_       = m;
  cap_     = std::min(m, kSteps);
  vectors_ = vectors;
  state_.resize(bytes_for(m, vectors));
  if (cluster() > 8) allow_large_clusters();
  wide_.resize(n_ > kWideFrom ? sizeof(double) * kWideStride * std::min(vectors, kWideVectors) : 0);
  if (!mail_) mail_ = static_cast<GmresMail *>(pinned_alloc(sizeof(GmresMail)));
}

void Arnoldi::reserve(int nb, int64_t steps, cudaStream_t s) {
  if (steps <= cap_) return;
  const int64_t cap = std::min(m_, std::max(steps, 2 * cap_));
  DeviceBuffer  next(stride(cap) * vectors_ * sizeof(double));
  for (int k = 0; k < nb; k++) {
    const StateView from(state_.as<double>() + k * stride(cap_), cap_), to(next.as<double>() + k * stride(cap), cap);
    auto            copy = [&](void *dst, const void *src, int64_t n) {
      MPIR_CUDA(cudaMemcpyAsync(dst, src, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
    };
    copy(to.ctl, from.ctl, from.R - reinterpret_cast<double *>(from.ctl));
    copy(to.R, from.R, cap_ * (cap_ + 1) / 2);
    copy(to.c, from.c, cap_);
    copy(to.s, from.s, cap_);
    copy(to.g, from.g, cap_ + 1);
  }
  MPIR_CUDA(cudaStreamSynchronize(s));
  state_ = std::move(next);
  cap_   = cap;
}

const int32_t *Arnoldi::active() const {
  return reinterpret_cast<const int32_t *>(state_.as<char>() + offsetof(GmresCtl, active));
}

// One CTA up to the entries its registers hold; 8 CTAs; 16 where that keeps
// the vector in registers or nearly so.
int Arnoldi::cluster() const {
  constexpr int64_t cta = static_cast<int64_t>(kThreads) * kRegs;
  return n_ <= cta ? 1 : n_ <= 8 * cta ? 8 : 16;
}

bool Arnoldi::wide(int nb) const { return n_ > kWideFrom && nb <= kWideVectors; }

void Arnoldi::begin(int nb, uint32_t act, const double *b, const VecFactors &fac, double *V, double tol,
                    cudaStream_t s) {
  const ArnoldiArgs a = make_args(n_, m_, cap_, stride(cap_), V, 0, state_.as<double>(), tol, mail_,
                                  wide(nb) ? wide_.as<double>() : nullptr);
  if (a.wide)
    launch_chained(0, k_wide_norm, 1, dim3(kWideCtas, nb, 1), kThreads, 0, s, a, act, b, fac);
  launch_chained(n_, a.wide ? k_gmres_begin<true> : k_gmres_begin<false>, cluster(), dim3(cluster(), nb, 1), kThreads, 0, s, a, act, b, fac);
}

void Arnoldi::first(int nb, double *V, double tol, cudaStream_t s) {
  const ArnoldiArgs a = make_args(n_, m_, cap_, stride(cap_), V, 0, state_.as<double>(), tol, mail_,
                                  wide(nb) ? wide_.as<double>() : nullptr);
  if (a.wide)
    launch_chained(0, k_wide_norm, 1, dim3(kWideCtas, nb, 1), kThreads, 0, s, a, 0u, nullptr, VecFactors{});
  launch_chained(n_, a.wide ? k_gmres_first<true> : k_gmres_first<false>, cluster(), dim3(cluster(), nb, 1), kThreads, 0, s, a);
  if (a.wide) launch_chained(0, k_wide_scale, 1, dim3(kWideCtas, nb, 1), kThreads, 0, s, a, 0);
}

void Arnoldi::step(int nb, int64_t j, double *V, int64_t block, double tol, cudaStream_t s) {
  const ArnoldiArgs a = make_args(n_, m_, cap_, stride(cap_), V, block, state_.as<double>(), tol, mail_,
                                  wide(nb) ? wide_.as<double>() : nullptr);
  if (a.wide)
    for (int64_t q = 0; q <= j + 1; q++)
      launch_chained(0, k_wide_sweep, 1, dim3(kWideCtas, nb, 1), kThreads, 0, s, a, j, q);
  launch_chained(n_, a.wide ? k_gmres_step<true> : k_gmres_step<false>, cluster(), dim3(cluster(), nb, 1), kThreads, 0, s, a, j);
  if (a.wide) launch_chained(0, k_wide_scale, 1, dim3(kWideCtas, nb, 1), kThreads, 0, s, a, j + 1);
}

void Arnoldi::end(int nb, uint32_t act, const double *V, int64_t block, double *x, bool update,
                  const VecFactors &scale, unsigned long long *inf, cudaStream_t s) {
  const ArnoldiArgs a = make_args(n_, m_, cap_, stride(cap_), const_cast<double *>(V), block, state_.as<double>(), 0.0, mail_,
                                  wide(nb) ? wide_.as<double>() : nullptr);
  launch_chained(n_, a.wide ? k_gmres_end<true> : k_gmres_end<false>, cluster(), dim3(cluster(), nb, 1), kThreads, 0, s, a, act, x, update ? 1 : 0,
                 scale, inf);
  if (a.wide)
    launch_chained(0, k_wide_end, 1, dim3(kWideCtas, nb, 1), kThreads, 0, s, a, act, x, update ? 1 : 0, scale, inf);
}

}  // namespace mpir
