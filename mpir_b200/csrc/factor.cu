// Numeric multifrontal LDL^T factorization on the GPU.
//
// The factor of P K P^T equals, entry for entry up to rounding, the one
// QDLDL_factor computes row by row (qdldl.hpp:172-345); it is organised here
// as a level-scheduled multifrontal method over the supernodal elimination
// tree instead:
//   * the scaled entries of K are scattered into zeroed panels;
//   * level by level (leaves first), each front gathers its children's
//     update matrices (extend-add), eliminates its own columns with a dense
//     partial LDL^T and leaves its Schur complement as its update matrix;
//   * fronts of at most kSmallFront rows are done whole in shared memory, one
//     thread block each; larger fronts go through a blocked right-looking
//     partial factorization whose steps are batched over all fronts of the
//     level: diagonal-block factor + inverse, a GEMM-shaped panel solve
//     (W = F L^{-T}, L = W D^{-1}) and a GEMM-shaped trailing update
//     C -= (L D) L^T.
// D is left on each panel's diagonal and copied to D / Dinv (permuted order).
#include <atomic>
#include <chrono>

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <string>

#include "common.cuh"
#include "engine.hpp"

namespace mpir {

// ---------------------------------------------------------------------------
// Scaling and assembly of K's entries.

// AD_i = 1/sqrt|k_ii| when |k_ii| > eps(UF), else 1 (gmres_ir.hpp:347-356).
__global__ void k_scaling(int64_t n, const int64_t *diag_pos, const double *Ax,
                          double eps, double *AD) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  double        d = 1.0;
  const int64_t p = diag_pos[i];
  if (p >= 0) {
    const double a = fabs(Ax[p]);
    if (a > eps) d = 1.0 / sqrt(a);
  }
  AD[i] = d;
}

// a_rc *= AD_r AD_c (gmres_ir.hpp:358-363) and scatter into the panels in the
// factor type.
__global__ void k_scatter(int64_t nnz, const double *Ax, const double *AD,
                          const int32_t *arow, const int32_t *acol,
                          const int64_t *amap, double *Axs, float *panel) {
  const int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (p >= nnz) return;
  const double v = Ax[p] * (AD[arow[p]] * AD[acol[p]]);
  Axs[p]         = v;
  panel[amap[p]] = static_cast<float>(v);
}

// Values of the full symmetric CSR of P K P^T: scaled and original.
__global__ void k_csr_values(int64_t nnzf, const int64_t *Ksrc,
                             const double *Axs, const double *Ax, double *Kval,
                             double *Korig) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= nnzf) return;
  const int64_t p = Ksrc[e];
  Kval[e]         = Axs[p];
  Korig[e]        = Ax[p];
}

__device__ __forceinline__ void note_pivot(FactorStatus *st, int32_t col,
                                           float d, int *npos) {
  if (d == 0.0f) atomicMin(&st->zero_pivot, col);
  if (!isfinite(d)) st->nonfinite = 1;
  if (d > 0.0f) (*npos)++;
}

// ---------------------------------------------------------------------------
// Small fronts: whole front in shared memory, a warp on every eighth column
// (lane = row, and row + 32), one barrier a pivot: a pivot's update reads its
// column as it stands, and the columns are scaled when they are written.  What
// bounds it is the chain of pivots; with the update spread over its entries by
// division of the thread's number and two barriers a pivot, a front of 64 rows
// took 37 us, 20 us so (both from a launch on, cold).
template <int HMAX>
__global__ void __launch_bounds__(kSmallThreads)
    k_small_fronts(const int32_t *list, const int64_t *sfirst,
                   const int64_t *srowptr, const int64_t *slofs,
                   const int64_t *uofs, const int64_t *child_ptr,
                   const int32_t *child_list, const int32_t *srel,
                   float *panel, float *uarena, float *D, float *Dinv,
                   FactorStatus *st) {
  static_assert(HMAX == 64 && kSmallThreads % 32 == 0, "rows by lane");
  constexpr int    kW = kSmallThreads / 32;
  __shared__ float F[HMAX][HMAX + 1];
  __shared__ float dinv_s[HMAX];
  const int        J    = list[blockIdx.x];
  const int        tid  = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int64_t    f    = sfirst[J];
  const int        w    = static_cast<int>(sfirst[J + 1] - f);
  const int        h    = static_cast<int>(srowptr[J + 1] - srowptr[J]);
  float           *P    = panel + slofs[J];
  for (int j = warp; j < h; j += kW)
    for (int i = lane; i < h; i += 32) F[i][j] = (j < w && i >= j) ? P[i + (int64_t)j * h] : 0.0f;
  __syncthreads();
  for (int64_t c = child_ptr[J]; c < child_ptr[J + 1]; c++) {
    const int      C  = child_list[c];
    const int      wc = static_cast<int>(sfirst[C + 1] - sfirst[C]);
    const int      rc = static_cast<int>(srowptr[C + 1] - srowptr[C]) - wc;
    const float   *U  = uarena + uofs[C];
    const int32_t *rl = srel + srowptr[C] + wc;
    // (a child's rows are among the front's: rc <= h; two of the warp's columns
    // are loaded before the first is added)
    const int     r0 = lane < rc ? rl[lane] : 0, r1 = lane + 32 < rc ? rl[lane + 32] : 0;
    constexpr int kCols = 2;
    for (int b0 = warp; b0 < rc; b0 += kCols * kW) {
      int   rb[kCols];
      float u0[kCols], u1[kCols];
#pragma unroll
      for (int q = 0; q < kCols; q++) {
        const int    b  = b0 + q * kW;
        const float *Ub = U + (int64_t)b * rc;
        rb[q] = b < rc ? rl[b] : 0;
        u0[q] = lane >= b && lane < rc ? Ub[lane] : 0.0f;
        u1[q] = lane + 32 >= b && lane + 32 < rc ? Ub[lane + 32] : 0.0f;
      }
#pragma unroll
      for (int q = 0; q < kCols; q++) {
        const int b = b0 + q * kW;
        if (lane >= b && lane < rc) F[r0][rb[q]] += u0[q];
        if (lane + 32 >= b && lane + 32 < rc) F[r1][rb[q]] += u1[q];
      }
    }
    __syncthreads();
  }
  int npos = 0;
  for (int k = 0; k < w; k++) {
    const float dk   = F[k][k];
    const float dinv = 1.0f / dk;
    const int   i1   = lane + 32;
    const float l0   = lane > k && lane < h ? F[lane][k] * dinv : 0.0f;
    const float l1   = i1 > k && i1 < h ? F[i1][k] * dinv : 0.0f;
    // columns k + 1 + .. of this warp
    for (int j = k + 1 + (warp + kW - (k + 1) % kW) % kW; j < h; j += kW) {
      const float fj = F[j][k];
      if (lane >= j && lane < h) F[lane][j] -= l0 * fj;
      if (i1 >= j && i1 < h) F[i1][j] -= l1 * fj;
    }
    if (tid == 0) {
      dinv_s[k]   = dinv;
      D[f + k]    = dk;
      Dinv[f + k] = dinv;
      note_pivot(st, static_cast<int32_t>(f + k), dk, &npos);
    }
    __syncthreads();
  }
  if (tid == 0) atomicAdd(&st->npos, npos);
  for (int j = warp; j < w; j += kW) {
    const float s = dinv_s[j];
    for (int i = lane; i < h; i += 32)
      if (i >= j) P[i + (int64_t)j * h] = i == j ? F[i][j] : F[i][j] * s;
  }
  const int r = h - w;
  if (r > 0) {
    float *U = uarena + uofs[J];
    for (int b = warp; b < r; b += kW)
      for (int a = lane; a < r; a += 32)
        U[a + (int64_t)b * r] = a >= b ? F[w + a][w + b] : 0.0f;
  }
}

// ---------------------------------------------------------------------------
// Extend-add of the children's update matrices into a level's large parents,
// one CTA per chunk of at most kEaChunk parent columns (EaChunk): the
// children that add to those columns, in child order with a barrier between
// them (siblings may add to the same entries), each child's columns of the
// chunk by all threads over the child's rows.  Every parent entry receives
// its children's contributions in child order.  Within a child each thread
// takes one row at a time across the chunk's columns: the row map entry is
// loaded one row ahead and all values of U_C and of the parent are loaded
// before any store (the source and the destination may both lie in the
// update arena, so the compiler would not reorder them itself).
// Where a launch has few chunks (the wide fronts' panels: 50 of 5,000 rows
// took 27 us on a third of the chip, 11 us split) a chunk's parent rows are
// split over gridDim.y CTAs, each of which finds its rows of a child by a
// 32-way search.  The others are bound by the bytes in flight: 48 registers
// for five CTAs an SM (three with 80 registers: 6.9 TB/s of L2 traffic; six
// spill), the children's descriptions kEaHits at a time in two round trips.
// A factorization's extend-adds: 1.04 -> 0.86 ms at n = 24,603, 15.0 -> 13.4 ms
// at n = 138,240.
constexpr int kEaHits = 16;

// First index a in [lo, lo + len) with rl[a] >= row (the end if none).
__device__ __forceinline__ int first_row(const int32_t *rl, int lo, int len, int row) {
  const int lane = threadIdx.x % 32;
  while (len > 0) {
    const int step = (len + 31) / 32, idx = (lane + 1) * step - 1;
    const int c    = __popc(__ballot_sync(0xffffffffu, idx < len && rl[lo + idx] < row));
    lo += c * step;
    if (step == 1) break;
    len = min(step - 1, len - c * step);
  }
  return lo;
}

__global__ void __launch_bounds__(256, 5)
    k_extend_add(const EaChunk *chunks, const EaHit *hits, const EaTask *tasks,
                 const int32_t *srel, float *panel, float *uarena) {
  __shared__ int64_t s_u[kEaHits], s_rel[kEaHits];
  __shared__ int     s_rc[kEaHits], s_lo[kEaHits], s_hi[kEaHits], s_a[2][kEaHits];
  const EaChunk ck   = chunks[blockIdx.x];
  const int     tid  = threadIdx.x, parts = gridDim.y, part = blockIdx.y;
  const bool    in_u = ck.c0 >= ck.wp;
  // Parent entry (row ra, column cb) at base + (cb - cbase) * ld + ra: in the
  // panel (rows from 0) or in the update matrix (rows from wp).
  float *const  base  = in_u ? uarena + ck.parent_u - ck.wp : panel + ck.parent_panel;
  const int64_t ld    = in_u ? ck.hp - ck.wp : ck.hp;
  const int     cbase = in_u ? ck.wp : 0;
  for (int h0 = ck.hit0; h0 < ck.hit1; h0 += kEaHits) {
    const int nh = min(kEaHits, ck.hit1 - h0);
    if (tid < nh) {
      const EaHit  hit = hits[h0 + tid];
      const EaTask tk  = tasks[hit.task];
      s_u[tid]    = tk.child_u;
      s_rel[tid]  = tk.rel;
      s_rc[tid]   = tk.rc;
      s_lo[tid]   = hit.ulo;
      s_hi[tid]   = hit.uhi;
      s_a[0][tid] = hit.ulo;
      s_a[1][tid] = tk.rc;
    }
    __syncthreads();
    if (parts > 1) {  // this part's parent rows
      const int rows = (ck.hp - ck.c0 + parts - 1) / parts;
      for (int e = tid / 32; e < 2 * nh; e += blockDim.x / 32) {
        const int q = e / 2, p = part + e % 2;
        if (p == 0 || p == parts) continue;
        const int a = first_row(srel + s_rel[q], s_lo[q], s_rc[q] - s_lo[q], ck.c0 + p * rows);
        if (tid % 32 == 0) s_a[e % 2][q] = a;
      }
      __syncthreads();
    }
    for (int q = 0; q < nh; q++) {
      const int32_t *rl = srel + s_rel[q];
      const float   *U  = uarena + s_u[q];
      const int      rc = s_rc[q], u0 = s_lo[q], nb = s_hi[q] - u0, end = s_a[1][q];
      float         *dst[kEaChunk];
      int            a  = s_a[0][q] + tid;
      int            ra = a < end ? rl[a] : 0;
#pragma unroll
      for (int u = 0; u < kEaChunk; u++)
        dst[u] = base + static_cast<int64_t>((u < nb ? rl[u0 + u] : cbase) - cbase) * ld;
      for (; a < end; a += blockDim.x) {
        const int an     = a + blockDim.x;
        const int ra_nxt = an < end ? rl[an] : 0;
        float     v[kEaChunk], o[kEaChunk];
#pragma unroll
        for (int u = 0; u < kEaChunk; u++) {
          const bool ok = u < nb && a >= u0 + u;
          v[u]          = ok ? U[a + static_cast<int64_t>(u0 + u) * rc] : 0.0f;
          o[u]          = ok ? dst[u][ra] : 0.0f;
        }
#pragma unroll
        for (int u = 0; u < kEaChunk; u++)
          if (u < nb && a >= u0 + u) dst[u][ra] = o[u] + v[u];
        ra = ra_nxt;
      }
      __syncthreads();
    }
  }
}

// ---------------------------------------------------------------------------
// Diagonal block of one step: LDL^T of the nbk x nbk block (nbk <= 128) and
// the inverse X = L^{-1} of its unit-lower factor, right-looking by panels of
// 32 columns in shared memory (row-major copies of the block and of X; the
// block is padded with a unit diagonal up to a multiple of 32).  Panel p:
//   A. warp 0 factors the 32 x 32 diagonal block (lane = row).  Its chain is
//      one broadcast, one reciprocal (the fast approximate one; D^{-1} itself
//      is the correctly rounded 1 / d_k), one product and one update a pivot;
//      the rest of a pivot's update takes the column from shared memory one
//      pivot later.  Every 8 pivots it signals a named barrier, and a warp
//      forms X_pp (lane = column) from them while it goes on; up to two more
//      follow that one with the rows below, eight columns at a time
//      (G = F X_pp^T = L D, kept transposed, then L = G D^{-1}).  The other twelve warps do
//      what the chain does not wait for, in 32 x 32 block products: the previous panel's update of the columns beyond this
//      panel, X_{p-1,b} = -X_{p-1,p-1} T_{p-1,b}, the contributions
//      T_ib += L_{i,p-1} X_{p-1,b} to the rows of X still to come (kept where
//      X_ib will be), and the stores of what is final (in panel 0 they read
//      the later panels' columns);
//   B. the next panel's columns take this panel's update.
// What bounds it: the chain of 128 pivots, and beside it the 128 bytes a cycle
// that shared memory returns to registers (a broadcast value costs a warp as
// much as 32 different ones), hence two rows a lane below the diagonal block
// and 4 x 4 values a lane in the products.  A block of 128 columns takes 29.8
// us, 35.0 with X_pp and G formed after the diagonal block and everything
// written at the end (32 columns 10 us both); the sums run in the same order as
// there.  Two pivots a turn: no gain.  Rows below by substitution beside the pivots
// instead of through X_pp: 28.4 us, but L moves by as much as its own error (2e-7)
// so, which the QDLDL functions pass on to their solution.
constexpr int kDiagLD = kNB + 4;  // Fs, Xs row stride (16-byte rows, lane = row conflict-free)
constexpr int kDiagSmemFloats = 2 * kNB * kDiagLD + 2 * 32 * kNB + 32 * 32;

__device__ __forceinline__ void bar_arrive(int id, int threads) {
  __threadfence_block();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_wait(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Row r of 32 values starting at a 16-byte boundary.
__device__ __forceinline__ void load_row32(float (&a)[32], const float *p) {
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const float4 v = reinterpret_cast<const float4 *>(p)[q];
    a[4 * q]     = v.x;
    a[4 * q + 1] = v.y;
    a[4 * q + 2] = v.z;
    a[4 * q + 3] = v.w;
  }
}
__device__ __forceinline__ void store_quad(float *p, float x, float y, float z, float w) {
  *reinterpret_cast<float4 *>(p) = make_float4(x, y, z, w);
}
// a[j] -= l col[j] for j > K of 32 (col: a broadcast row of shared memory).
template <int K>
__device__ __forceinline__ void update_row32(float (&a)[32], float l, const float *col) {
#pragma unroll
  for (int q = (K + 1) / 4; q < 8; q++) {
    const float4 v = reinterpret_cast<const float4 *>(col)[q];
    const float  f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (4 * q + u > K) a[4 * q + u] -= l * f[u];
  }
}
// f(integral constant k) for k = K0 .. K0 + 7.
template <int K>
struct Int {
  static constexpr int v = K;
};
template <int K0, class F>
__device__ __forceinline__ void each8(F f) {
  f(Int<K0>{});
  f(Int<K0 + 1>{});
  f(Int<K0 + 2>{});
  f(Int<K0 + 3>{});
  f(Int<K0 + 4>{});
  f(Int<K0 + 5>{});
  f(Int<K0 + 6>{});
  f(Int<K0 + 7>{});
}

// Phase A of panel p for warp 0: the diagonal block at (c0, c0).  Column k goes
// to Gt (unscaled, at row c0 + lane) and Ld (scaled).  The broadcasts that the
// next pivot waits for are issued before the loads of this one's column.  The
// updates' roundings are written out, whatever a compiler would fuse.  Pivot 0's
// update of column 30 alone is rounded twice, which is no better, but how
// factors have been rounded so far: with one rounding the QDLDL functions'
// unrefined solution moved by up to 5e-7 on one value set in five, at the same
// distance from float64.  Kept out of line: inlined into the kernel, whose
// other phases hold many registers, its chain of shuffles is scheduled about 1.5x
// slower.
__device__ __noinline__ void diag_panel(float *Fs, float *Gt, float *Ld, int c0, int n,
                                        const StepDesc &d, float *D, float *Dinv, float *packd,
                                        float *packs, FactorStatus *st, int &npos) {
  constexpr unsigned full = 0xffffffffu;
  const int          lane = threadIdx.x % 32, r = c0 + lane;
  float             *g = Gt + c0;
  float              a[32], fp[32], lp = 0.0f, piv = 1.0f;
  load_row32(a, Fs + r * kDiagLD + c0);
  float dk = __shfl_sync(full, a[0], 0), f1 = __shfl_sync(full, a[0], 1);
  g[lane] = a[0];
#pragma unroll
  for (int k = 0; k < 32; k++) {
    const float dv = __fdividef(1.0f, dk);
    if (k > 0) {  // the previous pivot's update of the columns beyond k
#pragma unroll
      for (int j = 0; j < 32; j++)
        if (j > k)
          a[j] = k == 1 && j == 30 ? __fsub_rn(a[j], __fmul_rn(lp, fp[j])) : __fmaf_rn(-lp, fp[j], a[j]);
    }
    if (lane == k) piv = dk;
    const float l = a[k] * dv;  // L[r][k]
    if (k < 31) {
      a[k + 1] -= l * f1;
      dk = __shfl_sync(full, a[k + 1], k + 1);
      if (k < 30) f1 = __shfl_sync(full, a[k + 1], k + 2);
      g[(k + 1) * kNB + lane] = a[k + 1];
    }
    Ld[32 * k + lane] = l;
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; q++)
      if (4 * q + 3 > k + 1) {
        const float4 v = *reinterpret_cast<const float4 *>(g + k * kNB + 4 * q);
        fp[4 * q]     = v.x;
        fp[4 * q + 1] = v.y;
        fp[4 * q + 2] = v.z;
        fp[4 * q + 3] = v.w;
      }
    lp = l;
    if (lane > k) a[k] = l;
    if (k % 8 == 7) bar_arrive(1 + k / 8, 64);
  }
#pragma unroll
  for (int q = 0; q < 8; q++)
    store_quad(Fs + r * kDiagLD + c0 + 4 * q, a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
  if (r < n) {
    const float   pinv = 1.0f / piv;
    const int64_t cidx = (int64_t)d.col0 + d.kb + r;
    D[cidx]            = piv;
    Dinv[cidx]         = pinv;
    if (packd != nullptr && d.pd >= 0) {
      packd[d.pd + d.kb + r] = piv;
      packs[d.pd + d.kb + r] = copysignf(sqrtf(fabsf(piv)), piv);
    }
    note_pivot(st, static_cast<int32_t>(cidx), piv, &npos);
  }
}

// Phase A for R x 32 rows below the diagonal block (lane = rows r, r + 32, ..):
// G = F X_pp^T, L = G D^{-1}, eight columns (rows of X_pp) at a time as the
// inverse's warp finishes them.
template <int R>
__device__ __noinline__ void diag_rows(float *Fs, float *Gt, const float *Xpp, int c0, int nsync, int r) {
  const float *g   = Gt + c0;
  const int    l8  = threadIdx.x % 8;
  float       *row = Fs + r * kDiagLD + c0;
  float        f[R][32], out[R][8];
#pragma unroll
  for (int v = 0; v < R; v++) load_row32(f[v], row + 32 * v * kDiagLD);
  auto column = [&](auto jc) {
    constexpr int j = decltype(jc)::v;
    float         acc[R];
#pragma unroll
    for (int v = 0; v < R; v++) acc[v] = 0.0f;
#pragma unroll
    for (int q = 0; q <= j / 4; q++) {  // row j of X_pp is zero right of j
      const float4 x = reinterpret_cast<const float4 *>(Xpp + j * kDiagLD)[q];
#pragma unroll
      for (int v = 0; v < R; v++) {
        acc[v] += f[v][4 * q] * x.x;
        acc[v] += f[v][4 * q + 1] * x.y;
        acc[v] += f[v][4 * q + 2] * x.z;
        acc[v] += f[v][4 * q + 3] * x.w;
      }
    }
#pragma unroll
    for (int v = 0; v < R; v++) {
      Gt[j * kNB + r + 32 * v] = acc[v];
      out[v][j % 8]            = acc[v];
    }
  };
  // L of 8 columns (lane l8 of each 8 divides for column k0 + l8).
  auto finish = [&](int k0) {
    const float pv = 1.0f / g[(k0 + l8) * kNB + k0 + l8];
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const float pk = __shfl_sync(0xffffffffu, pv, u, 8);
#pragma unroll
      for (int v = 0; v < R; v++) out[v][u] *= pk;
    }
#pragma unroll
    for (int v = 0; v < R; v++) {
      float *p = row + 32 * v * kDiagLD + k0;
      store_quad(p, out[v][0], out[v][1], out[v][2], out[v][3]);
      store_quad(p + 4, out[v][4], out[v][5], out[v][6], out[v][7]);
    }
  };
  bar_wait(6, nsync);
  each8<0>(column);
  finish(0);
  bar_wait(7, nsync);
  each8<8>(column);
  finish(8);
  bar_wait(8, nsync);
  each8<16>(column);
  finish(16);
  bar_wait(9, nsync);
  each8<24>(column);
  finish(24);
}

// Phase A for X of the diagonal block (lane = column): x = L^{-1} e_lane.  Row k
// is final at pivot k; nsync: threads of the barriers that hand eight rows on.
__device__ __noinline__ void diag_inverse(float *Xpp, const float *Ld, int nsync) {
  const int lane = threadIdx.x % 32;
  float     x[32];
#pragma unroll
  for (int i = 0; i < 32; i++) x[i] = i == lane ? 1.0f : 0.0f;
  auto step = [&](auto kk) {
    constexpr int k         = decltype(kk)::v;
    Xpp[k * kDiagLD + lane] = x[k];
    update_row32<k>(x, x[k], Ld + 32 * k);
  };
  bar_wait(1, 64);
  each8<0>(step);
  if (nsync > 32) bar_arrive(6, nsync);
  bar_wait(2, 64);
  each8<8>(step);
  if (nsync > 32) bar_arrive(7, nsync);
  bar_wait(3, 64);
  each8<16>(step);
  if (nsync > 32) bar_arrive(8, nsync);
  bar_wait(4, 64);
  each8<24>(step);
  if (nsync > 32) bar_arrive(9, nsync);
}

// Half of a 32 x 32 block product: 16 columns (half 0 or 1) by one warp, a lane
// 4 x 4.  kSub: C -= A B.  kFirst, kNext: C = A B, C += A B, one sum over both.
// kNeg: C = -A B in four sums (terms k mod 4); C may be B.
enum DiagMode { kSub, kFirst, kNext, kNeg };
template <DiagMode MODE>
__device__ __noinline__ void diag_product(const float *A, const float *B, int ldb, float *C, int half) {
  constexpr int LD = kDiagLD, S = MODE == kNeg ? 4 : 1;
  const int     lane = threadIdx.x % 32, i0 = 4 * (lane / 4), j0 = 16 * half + 4 * (lane % 4);
  float         acc[S][4][4] = {};
  A += i0 * LD;
  B += j0;
  C += i0 * LD + j0;
  if (MODE == kNext) {
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const float4 o = *reinterpret_cast<const float4 *>(C + r * LD);
      acc[0][r][0] = o.x;
      acc[0][r][1] = o.y;
      acc[0][r][2] = o.z;
      acc[0][r][3] = o.w;
    }
  }
#pragma unroll 2
  for (int k = 0; k < 32; k += 4) {
    float4 b[4];
#pragma unroll
    for (int u = 0; u < 4; u++) b[u] = *reinterpret_cast<const float4 *>(B + (k + u) * ldb);
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const float4 f = *reinterpret_cast<const float4 *>(A + r * LD + k);
      const float  a[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
      for (int u = 0; u < 4; u++) {
        acc[u % S][r][0] += a[u] * b[u].x;
        acc[u % S][r][1] += a[u] * b[u].y;
        acc[u % S][r][2] += a[u] * b[u].z;
        acc[u % S][r][3] += a[u] * b[u].w;
      }
    }
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < 4; r++) {
    float o[4];
#pragma unroll
    for (int s = 0; s < 4; s++)
      o[s] = MODE == kNeg ? -((acc[0][r][s] + acc[1 % S][r][s]) + (acc[2 % S][r][s] + acc[3 % S][r][s]))
                          : acc[0][r][s];
    if (MODE == kSub) {
      const float4 c = *reinterpret_cast<const float4 *>(C + r * LD);
      o[0] = c.x - o[0];
      o[1] = c.y - o[1];
      o[2] = c.z - o[2];
      o[3] = c.w - o[3];
    }
    store_quad(C + r * LD, o[0], o[1], o[2], o[3]);
  }
}

// Panel p's columns into the front (P, column stride h, n rows), by warp u of
// nu: 4 columns a turn, lane = row.
__device__ __noinline__ void diag_store_panel(float *P, int64_t h, int n, int nblk, const float *Fs, int p,
                                              int u, int nu) {
  const int lane = threadIdx.x % 32, cnt = 8 * (nblk - p);
#pragma unroll 2
  for (int e = u; e < cnt; e += nu) {
    const int    i = 32 * (p + e / 8) + lane, j = 32 * p + 4 * (e % 8);
    const float4 v = *reinterpret_cast<const float4 *>(Fs + i * kDiagLD + j);
    float       *q = P + i + (int64_t)j * h;
    const int    k = i < n ? i - j : -1;
    if (k >= 0) q[0] = v.x;
    if (k >= 1) q[h] = v.y;
    if (k >= 2) q[2 * h] = v.z;
    if (k >= 3) q[3 * h] = v.w;
  }
}
// Row block x of X into Lv (blocks above the diagonal blocks, rows and columns
// of the pad are zero), by warp u of nu.
__device__ __noinline__ void diag_store_x(float *Lv, int n, int n32, const float *Xs, int x, int u, int nu) {
  const int i = 32 * x + threadIdx.x % 32;
#pragma unroll 2
  for (int e = u; e < n32 / 4; e += nu) {
    const int j = 4 * e, k = j < 32 * (x + 1) && i < n ? n - j : 0;
    float4    v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (k > 0) v = *reinterpret_cast<const float4 *>(Xs + i * kDiagLD + j);
    float *q   = Lv + i + j * kNB;
    q[0]       = k > 0 ? v.x : 0.0f;
    q[kNB]     = k > 1 ? v.y : 0.0f;
    q[2 * kNB] = k > 2 ? v.z : 0.0f;
    q[3 * kNB] = k > 3 ? v.w : 0.0f;
  }
}

__global__ void __launch_bounds__(kDiagThreads)
    k_diag_block(const StepDesc *descs, float *panel, float *linv, float *D, float *Dinv,
                 float *packd, float *packs, FactorStatus *st) {
  static_assert(kDiagThreads == 4 * kNB, "diag kernel thread mapping");
  constexpr int LD = kDiagLD;
  extern __shared__ __align__(16) float sm[];
  float          *Fs = sm;                 // the block, row-major
  float          *Xs = Fs + kNB * LD;      // X, row-major
  float          *G2 = Xs + kNB * LD;      // G^T of two panels, by panel parity
  float          *Ld = G2 + 2 * 32 * kNB;  // L^T of the current diagonal block
  const StepDesc   d    = descs[blockIdx.x];
  const int        n    = d.nbk;
  const int        nblk = (n + 31) / 32, n32 = 32 * nblk;
  const int64_t    h    = d.h;
  const int        tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  float           *P = panel + d.panel + d.kb + (int64_t)d.kb * h, *Lv = linv + d.linv;
  // Columns j .. j + 3 of row i (lower triangle, unit pad), as loads in flight.
  auto quad = [&](int i, int j) {
    const float *q  = P + i + (int64_t)j * h;
    auto         at = [&](int u) {
      return i >= j + u && i < n ? q[u * h] : (i == j + u ? 1.0f : 0.0f);
    };
    return make_float4(at(0), at(1), at(2), at(3));
  };
  {
    const int i = tid % kNB, c = tid / kNB;
    if (i < n32) {
      const float4 v0 = quad(i, 4 * c), v1 = quad(i, 16 + 4 * c);
      *reinterpret_cast<float4 *>(Fs + i * LD + 4 * c)      = v0;
      *reinterpret_cast<float4 *>(Fs + i * LD + 16 + 4 * c) = v1;
    } else {  // rows of X beyond the block
      for (int j = c; j < n32; j += 4) Lv[i + j * kNB] = 0.0f;
    }
  }
  __syncthreads();
  int npos = 0;
  for (int p = 0;; p++) {
    const int c0 = 32 * p, rest = nblk - 1 - p, nsync = 32 * (1 + (rest + 1) / 2);
    float    *Gt = G2 + (p & 1) * 32 * kNB, *Xpp = Xs + c0 * LD + c0;
    // A.
    if (warp == 0) {
      diag_panel(Fs, Gt, Ld, c0, n, d, D, Dinv, packd, packs, st, npos);
    } else if (warp == 1) {
      if (rest >= 2)
        diag_rows<2>(Fs, Gt, Xpp, c0, nsync, c0 + 32 + lane);
      else if (rest == 1)
        diag_rows<1>(Fs, Gt, Xpp, c0, nsync, c0 + 32 + lane);
    } else if (warp == 2) {
      if (rest == 3) diag_rows<1>(Fs, Gt, Xpp, c0, nsync, c0 + 96 + lane);
    } else if (warp == 3) {
      diag_inverse(Xpp, Ld, nsync);
    } else {
      const int u = warp - 4, half = u % 2;
      if (p == 0) {
        // the later panels' columns: row blocks 1 .. nblk - 1, 8 quads a panel
        const int nq = 4 * nblk * (nblk - 1);
#pragma unroll 4
        for (int e = u; e < nq; e += 12) {
          const int b = e >= 24 ? 3 : e >= 8 ? 2 : 1, j = 32 + 4 * (e - 4 * b * (b - 1)), i = 32 * b + lane;
          *reinterpret_cast<float4 *>(Fs + i * LD + j) = quad(i, j);
        }
      } else {
        // Half a block product a warp: p - 1 of X_{p-1,b}; the update of blocks
        // (i, j), p < j <= i; T_{i,p-1}.  Then, with X_{p-1,b}, T_ib for b < p - 1.
        const int    q = p - 1, nd = rest * (rest + 1) / 2, w = u / 2;
        const float *Lq = Fs + 32 * q;  // L_{.,q}
        if (w < q) {
          float *X = Xs + 32 * q * LD + 32 * w;
          diag_product<kNeg>(Xs + 32 * q * LD + 32 * q, X, LD, X, half);
        } else if (w < q + nd) {
          const int e = w - q, i = p + 1 + (e >= 1) + (e >= 3), j = p + 1 + e - (i - p - 1) * (i - p) / 2;
          diag_product<kSub>(Lq + 32 * i * LD, G2 + (q & 1) * 32 * kNB + 32 * j, kNB,
                             Fs + 32 * i * LD + 32 * j, half);
        } else if (w < q + nd + rest + 1) {
          const int i = p + w - q - nd;
          diag_product<kFirst>(Lq + 32 * i * LD, Xs + 32 * q * LD + 32 * q, LD, Xs + 32 * i * LD + 32 * q,
                               half);
        }
        diag_store_panel(P, h, n, nblk, Fs, q, 11 - u, 12);
        bar_wait(5, 384);
        const int e = 5 - w;
        if (e < q * (rest + 1)) {
          const int i = p + e / q, b = e % q;
          diag_product<kNext>(Lq + 32 * i * LD, Xs + 32 * q * LD + 32 * b, LD, Xs + 32 * i * LD + 32 * b,
                              half);
        }
        diag_store_x(Lv, n, n32, Xs, q, u, 12);
      }
    }
    __syncthreads();
    if (rest == 0) break;
    // B.
    if (warp < 2 * rest) {
      const int i = c0 + 32 + 32 * (warp / 2);
      diag_product<kSub>(Fs + i * LD + c0, Gt + c0 + 32, kNB, Fs + i * LD + c0 + 32, warp % 2);
    }
    __syncthreads();
  }
  if (warp == 0) {
    npos = __reduce_add_sync(0xffffffffu, npos);
    if (tid == 0 && npos > 0) atomicAdd(&st->npos, npos);
  }
  const int last = nblk - 1;
  if (warp < 2 * last) {
    float *X = Xs + 32 * last * LD + 32 * (warp / 2);
    diag_product<kNeg>(Xs + 32 * last * LD + 32 * last, X, LD, X, warp % 2);
  }
  __syncthreads();
  diag_store_panel(P, h, n, nblk, Fs, last, warp, kDiagThreads / 32);
  diag_store_x(Lv, n, n32, Xs, last, kDiagThreads / 32 - 1 - warp, kDiagThreads / 32);
}

// ---------------------------------------------------------------------------
// GEMM-shaped kernels of a step (FP32 SIMT, 128x128 tiles, K in slices of 16).
//   TRSM:   C = (A B^T) .* dinv(cols), in place over A's block column;
//           A = panel rows below the block, B = Linv of the block.
//   UPDATE: C -= (A .* d(k)) B^T on the lower part; A = B = the eliminated
//           block column (rows below), C = trailing panel or update matrix.
constexpr int kBM = 128, kBN = 128, kBK = 16;

template <bool TRSM>
__global__ void __launch_bounds__(kGemmThreads)
    k_step_gemm(const StepDesc *descs, int ndesc, float *panel, float *uarena,
                const float *linv, const float *Dinv, float *pack) {
  // Two slices in shared memory: slice s+1 is loaded into registers while
  // slice s is multiplied, then stored into the other buffer.
  __shared__ float As[2][kBK][kBM];
  __shared__ float Bs[2][kBK][kBN];
  __shared__ float sd[kNB];
  const int        t  = blockIdx.x;
  int              lo = 0, hi = ndesc - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    const int t0  = TRSM ? descs[mid].trsm_tile0 : descs[mid].upd_tile0;
    if (t0 <= t) lo = mid; else hi = mid - 1;
  }
  const StepDesc d     = descs[lo];
  int            local = t - (TRSM ? d.trsm_tile0 : d.upd_tile0);
  const int64_t  h     = d.h;
  const int      kb = d.kb, nbk = d.nbk, w = d.w;
  const float   *A, *B;
  float         *C;
  int64_t        lda, ldb, ldc;
  int            M, N, m0, n0;
  const int      K = nbk;
  float         *Pp = panel + d.panel;
  if (TRSM) {
    M   = static_cast<int>(h) - kb - nbk;
    N   = nbk;
    A   = Pp + (kb + nbk) + (int64_t)kb * h;
    lda = h;
    B   = linv + d.linv;
    ldb = kNB;
    C   = Pp + (kb + nbk) + (int64_t)kb * h;
    ldc = h;
    m0  = local * kBM;
    n0  = 0;
  } else {
    if (local < d.upd_panel_tiles) {
      M = static_cast<int>(h) - kb - nbk;
      N = w - kb - nbk;
      A = Pp + (kb + nbk) + (int64_t)kb * h;
      C = Pp + (kb + nbk) + (int64_t)(kb + nbk) * h;
      ldc = h;
    } else {
      local -= d.upd_panel_tiles;
      M = N = static_cast<int>(h) - w;
      A     = Pp + w + (int64_t)kb * h;
      C     = uarena + d.uofs;
      ldc   = M;
    }
    lda = ldb = h;
    B         = A;
    const int ntr = (M + kBM - 1) / kBM;
    int       j   = 0;
    while (local >= ntr - j) {
      local -= ntr - j;
      j++;
    }
    m0 = (j + local) * kBM;
    n0 = j * kBN;
    for (int k = threadIdx.x; k < nbk; k += blockDim.x)
      sd[k] = Pp[(kb + k) + (int64_t)(kb + k) * h];
  }
  const int tid = threadIdx.x;
  const int tr = tid / 16, tc = tid % 16;
  float     acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) acc[i][j] = 0.0f;
  __syncthreads();
  constexpr int kLoads = (kBM * kBK) / kGemmThreads;
  float         ra[kLoads], rb[kLoads];
  auto          load = [&](int k0) {
#pragma unroll
    for (int q = 0; q < kLoads; q++) {
      const int idx = tid + q * kGemmThreads;
      const int i = idx % kBM, kk = idx / kBM;
      const int r = m0 + i, k = k0 + kk;
      float     v = 0.0f;
      if (r < M && k < K) {
        v = A[r + (int64_t)k * lda];
        if (!TRSM) v *= sd[k];
      }
      ra[q]       = v;
      const int c = n0 + i;
      rb[q]       = (c < N && k < K) ? B[c + (int64_t)k * ldb] : 0.0f;
    }
  };
  auto store = [&](int buf) {
#pragma unroll
    for (int q = 0; q < kLoads; q++) {
      const int idx = tid + q * kGemmThreads;
      As[buf][idx / kBM][idx % kBM] = ra[q];
      Bs[buf][idx / kBM][idx % kBM] = rb[q];
    }
  };
  load(0);
  store(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += kBK) {
    if (k0 + kBK < K) load(k0 + kBK);  // in flight during this slice
#pragma unroll
    for (int kk = 0; kk < kBK; kk++) {
      float a[8], b[8];
#pragma unroll
      for (int i = 0; i < 8; i++) a[i] = As[buf][kk][tr * 8 + i];
#pragma unroll
      for (int j = 0; j < 8; j++) b[j] = Bs[buf][kk][tc * 8 + j];
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    if (k0 + kBK < K) {
      store(buf ^ 1);
      __syncthreads();
      buf ^= 1;
    }
  }
  if (!TRSM) {
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int c = n0 + tc * 8 + j;
      if (c >= N) continue;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const int r = m0 + tr * 8 + i;
        if (r < M && r >= c) C[r + (int64_t)c * ldc] -= acc[i][j];
      }
    }
    return;
  }
  // TRSM epilogue: the tile times Dinv goes through shared memory, then to
  // the panel as 128-row column segments (one warp per column) and to the
  // packed front as whole 2 KB K-groups (PackedFront), both coalesced.
  extern __shared__ float tile_s[];  // kBM x (kBN + 1)
  constexpr int           LT = kBN + 1;
  float                   dvs[8];
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const int c = n0 + tc * 8 + j;
    dvs[j]      = c < N ? Dinv[(int64_t)d.col0 + kb + c] : 0.0f;
  }
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) tile_s[(tr * 8 + i) * LT + tc * 8 + j] = acc[i][j] * dvs[j];
  __syncthreads();
  const int warp = tid / 32, lane = tid % 32;
  for (int c = warp; c < N; c += kGemmThreads / 32)
#pragma unroll
    for (int q = 0; q < kBM / 32; q++) {
      const int r = lane + 32 * q;
      if (m0 + r < M) C[m0 + r + (int64_t)c * ldc] = tile_s[r * LT + c];
    }
  if (pack != nullptr && d.pk >= 0) {
    float *pk = pack + d.pk;
    for (int e = tid; e < kBM * (kBN / 4); e += kGemmThreads) {
      const int m = e % kBM, g = e / kBM, c0 = 4 * g;
      if (c0 >= N || m0 + m >= M) continue;
      const int rf = kb + nbk + m0 + m;  // row of the front
      const int p  = rf < w ? rf : rf - w + d.pk_wt;
      float4    v;
      v.x = tile_s[m * LT + c0 + 0];
      v.y = tile_s[m * LT + c0 + 1];
      v.z = tile_s[m * LT + c0 + 2];
      v.w = tile_s[m * LT + c0 + 3];
      *reinterpret_cast<float4 *>(pk +
                                  static_cast<int64_t>(p >> 7) * d.pk_g * PackedFront::kGroupFloats +
                                  static_cast<int64_t>((kb + c0) >> 2) * PackedFront::kGroupFloats +
                                  (p & 127) * 4) = v;
    }
  }
}

// ---------------------------------------------------------------------------
// GemmProb updates on the SIMT units (float32), the same tile and split
// mapping as the tensor-core kernel.
__device__ __forceinline__ void locate_tile(const GemmProb &pb, int local, int &sp, int &tile,
                                            int &m0, int &n0) {
  sp     = local % pb.splits;
  int tl = local / pb.splits;
  tile   = tl;
  int j  = 0;
  if (pb.lower) {
    while (tl >= pb.ntm - j) {
      tl -= pb.ntm - j;
      j++;
    }
    m0 = (j + tl) * kBM;
  } else {
    j  = tl / pb.ntm;
    m0 = (tl % pb.ntm) * kBM;
  }
  n0 = j * kBN;
}

__global__ void __launch_bounds__(kGemmThreads)
    k_gemm_simt(const GemmProb *probs, int nprob, float *panel, float *uarena, const float *D,
                float *ws) {
  __shared__ float As[kBK][kBM];
  __shared__ float Bs[kBK][kBN];
  const int        t  = blockIdx.x;
  int              lo = 0, hi = nprob - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (probs[mid].tile0 <= t) lo = mid; else hi = mid - 1;
  }
  const GemmProb pb = probs[lo];
  int            sp, tile, m0, n0;
  locate_tile(pb, t - pb.tile0, sp, tile, m0, n0);
  const int     M = pb.M, N = pb.N, K = pb.K;
  const int     ks   = ((K + pb.splits - 1) / pb.splits + 31) / 32 * 32;
  const int     k_lo = sp * ks, k_hi = min(K, k_lo + ks);
  const float  *A    = panel + pb.a_ofs;
  const int64_t lda  = pb.lda;
  const float  *Dk   = D + pb.d_ofs;
  const int     tid  = threadIdx.x;
  const int     tr = tid / 16, tc = tid % 16;
  float         acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; i++)
#pragma unroll
    for (int j = 0; j < 8; j++) acc[i][j] = 0.0f;
  for (int k0 = k_lo; k0 < k_hi; k0 += kBK) {
#pragma unroll
    for (int q = 0; q < (kBM * kBK) / kGemmThreads; q++) {
      const int idx = tid + q * kGemmThreads;
      const int i = idx % kBM, kk = idx / kBM;
      const int k = k0 + kk;
      const bool kin = k < k_hi;
      const int r = m0 + i < M ? gemm_out_row(pb, m0 + i) : -1, c = n0 + i;
      As[kk][i] = (r >= 0 && kin) ? A[r + (int64_t)k * lda] * Dk[k] : 0.0f;
      Bs[kk][i] = (c < N && kin) ? A[c + (int64_t)k * lda] : 0.0f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kBK; kk++) {
      float a[8], b[8];
#pragma unroll
      for (int i = 0; i < 8; i++) a[i] = As[kk][tr * 8 + i];
#pragma unroll
      for (int j = 0; j < 8; j++) b[j] = Bs[kk][tc * 8 + j];
#pragma unroll
      for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
  if (pb.splits > 1) {
    float *W = ws + pb.ws_ofs + (static_cast<int64_t>(tile) * pb.splits + sp) * (kBM * kBN);
#pragma unroll
    for (int j = 0; j < 8; j++)
#pragma unroll
      for (int i = 0; i < 8; i++) W[(tr * 8 + i) + (tc * 8 + j) * kBM] = acc[i][j];
    return;
  }
  float *C = (pb.c_in_u ? uarena : panel) + pb.c_ofs;
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const int c = n0 + tc * 8 + j;
    if (c >= N) continue;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int r = m0 + tr * 8 + i < M ? gemm_out_row(pb, m0 + tr * 8 + i) : -1;
      if (r >= 0 && (!pb.lower || r >= c))
        C[r + (int64_t)c * pb.ldc] = (pb.c_in_u ? 0.0f : C[r + (int64_t)c * pb.ldc]) - acc[i][j];
    }
  }
}

// C -= sum of the split partials of one tile, added in split order.  A tile
// is reduced by kReduceSlices CTAs, one float4 group (4 consecutive rows of a
// column) per thread: the late left-looking steps of a large front have a
// few tiles and many splits, so one CTA per tile would sum long chains
// alone.  The partials are loaded four splits at a time and added in order.
constexpr int kReduceSlices = 16;

__global__ void __launch_bounds__(256)
    k_split_reduce(const GemmProb *probs, int nprob, float *panel, float *uarena,
                   const float *ws) {
  static_assert(kBM * kBN / 4 == kReduceSlices * 256, "one float4 group per thread");
  const int t = blockIdx.x / kReduceSlices, slice = blockIdx.x % kReduceSlices;
  int       lo = 0, hi = nprob - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (probs[mid].rtile0 <= t) lo = mid; else hi = mid - 1;
  }
  const GemmProb pb = probs[lo];
  int            sp, tile, m0, n0;
  locate_tile(pb, (t - pb.rtile0) * pb.splits, sp, tile, m0, n0);
  float         *C  = (pb.c_in_u ? uarena : panel) + pb.c_ofs;
  const int      g  = slice * 256 + threadIdx.x;
  const float4  *W  = reinterpret_cast<const float4 *>(
                         ws + pb.ws_ofs + static_cast<int64_t>(tile) * pb.splits * (kBM * kBN)) + g;
  constexpr int  kT = kBM * kBN / 4;  // float4 groups of a tile
  float4         acc = make_float4(0.f, 0.f, 0.f, 0.f);
  int            q   = 0;
  for (; q + 4 <= pb.splits; q += 4) {
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = __ldcs(W + static_cast<int64_t>(q + u) * kT);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      acc.x += v[u].x;
      acc.y += v[u].y;
      acc.z += v[u].z;
      acc.w += v[u].w;
    }
  }
  for (; q < pb.splits; q++) {
    const float4 v = __ldcs(W + static_cast<int64_t>(q) * kT);
    acc.x += v.x;
    acc.y += v.y;
    acc.z += v.z;
    acc.w += v.w;
  }
  const int   e = 4 * g;
  const int   c = n0 + e / kBM;
  int64_t     at[4];
  float       cv[4];
  const float a[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
  for (int v = 0; v < 4; v++) {
    const int m = m0 + e % kBM + v;
    const int r = m < pb.M ? gemm_out_row(pb, m) : -1;
    at[v] = (r < 0 || c >= pb.N || (pb.lower && r < c)) ? -1 : r + (int64_t)c * pb.ldc;
    cv[v] = (!pb.c_in_u && at[v] >= 0) ? C[at[v]] : 0.0f;
  }
#pragma unroll
  for (int v = 0; v < 4; v++)
    if (at[v] >= 0) C[at[v]] = cv[v] - a[v];
}

// The panels rounded to bfloat16 (bf != 0) or float16 for the solves of the
// 16-bit tiers: L is stored in the tier's type and the solves read half the
// bytes (their arithmetic stays float64).
__global__ void k_panel_to16(int64_t n, const float *in, uint16_t *out, int bf) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    if (bf) {
      const __nv_bfloat16 v = __float2bfloat16_rn(in[i]);
      out[i]                = *reinterpret_cast<const uint16_t *>(&v);
    } else {
      const __half v = __float2half_rn(in[i]);
      out[i]         = *reinterpret_cast<const uint16_t *>(&v);
    }
  }
}

// ---------------------------------------------------------------------------
// Plan construction.

void Plan::build(Symbolic &&sym, cudaStream_t s, bool upload) {
  S              = std::move(sym);
  const int64_t ns = S.ns;
  nnz_full         = static_cast<int64_t>(S.Kj.size());
  // Persistent Linv storage for the large fronts.
  linv_elems   = 0;
  update_flops = 0;
  trsm_flops   = 0;
  pk_ofs.assign(ns, -1);
  pd_ofs.assign(ns, -1);
  pk_elems = pd_elems = 0;
  for (int64_t J = 0; J < ns; J++)
    if (is_large(J)) {
      pk_ofs[J] = pk_elems;
      pk_elems += pk_tiles(J) * pk_groups(J) * PackedFront::kGroupFloats;
      pd_ofs[J] = pd_elems;
      pd_elems += pk_groups(J) * 4;
    }
  // Per-level launch lists.
  levels.assign(S.nlevels, LevelPlan{});
  h_small.clear();
  h_large.clear();
  std::vector<StepDesc> descs;
  std::vector<EaTask>   tasks;
  std::vector<EaChunk>  chunks_h;
  std::vector<EaHit>    hits_h;
  std::vector<GemmProb> probs;
  ws_elems    = 0;
  bconv_elems = 0;
  // Tiles, K splits, launch offsets and workspace of the problems
  // [begin, begin + count) of one launch.  With fewer tiles than about two
  // per SM, K is split (at least 256 per split) and the partials reduced.
  auto finish_launch = [&](int32_t begin, int32_t count, int32_t &tiles, int32_t &rtiles,
                           int32_t &convs) {
    int64_t total = 0;
    for (int32_t q = begin; q < begin + count; q++) {
      GemmProb &g  = probs[q];
      g.ntm        = (g.M + kBM - 1) / kBM;
      const int nn = (g.N + kBN - 1) / kBN;
      g.ntiles     = g.lower ? nn * g.ntm - nn * (nn - 1) / 2 : nn * g.ntm;
      total += g.ntiles;
      const double Mr = g.M, Nc = g.N;
      update_flops += 2.0 * g.K * (g.lower ? Nc * Mr - Nc * (Nc - 1) / 2 : Nc * Mr);
    }
    // Splits of K: the count s (at least 256 of K per split) that minimises
    // waves(total tiles x s over the resident CTAs) x (K / s + a fixed cost
    // per CTA of about 128 columns of K); partial tiles are reduced after.
    const int64_t resident = static_cast<int64_t>(kSMs) * tc_ctas_per_sm();
    int64_t       kmax     = 0;
    for (int32_t q = begin; q < begin + count; q++) kmax = std::max<int64_t>(kmax, probs[q].K);
    int64_t best_s = 1;
    double  best_c = 1e300;
    for (int64_t sp = 1; sp <= std::max<int64_t>(1, kmax / 256); sp++) {
      const double waves = static_cast<double>((total * sp + resident - 1) / resident);
      const double c     = waves * (static_cast<double>((kmax + sp - 1) / sp) + 128.0);
      if (c < best_c - 1e-9) {
        best_c = c;
        best_s = sp;
      }
    }
    int64_t t0 = 0, r0 = 0, w0 = 0;
    for (int32_t q = begin; q < begin + count; q++) {
      GemmProb &g = probs[q];
      g.splits    = 1;
      const int64_t want = std::max<int64_t>(1, std::min<int64_t>(best_s, g.K / 256));
      if (want > 1) {
        // Split length as the kernels compute it (a multiple of 32); then as
        // many splits as that length needs, so no split is empty.
        const int64_t ks = ((g.K + want - 1) / want + 31) / 32 * 32;
        g.splits         = static_cast<int32_t>((g.K + ks - 1) / ks);
      }
      g.tile0  = static_cast<int32_t>(t0);
      t0 += static_cast<int64_t>(g.ntiles) * g.splits;
      g.rtile0 = static_cast<int32_t>(r0);
      g.ws_ofs = -1;
      if (g.splits > 1) {
        r0 += g.ntiles;
        g.ws_ofs = w0;
        w0 += static_cast<int64_t>(g.ntiles) * g.splits * kBM * kBN;
      }
    }
    tiles    = static_cast<int32_t>(t0);
    rtiles   = static_cast<int32_t>(r0);
    ws_elems = std::max(ws_elems, w0);
    // B converted once per launch for the 3xTF32 product: the problem's B
    // row tiles, all K-groups its K range reads.
    int64_t c0 = 0, b0 = 0;
    for (int32_t q = begin; q < begin + count; q++) {
      GemmProb &g = probs[q];
      g.btiles    = (g.N + kBN - 1) / kBN;
      g.bgroups   = static_cast<int32_t>((g.K + 31) / 32 * 8);
      g.bprow     = static_cast<int64_t>(g.bgroups) * PackedFront::kGroupFloats;
      g.bc        = b0;
      g.bc_lo     = b0 + g.btiles * g.bprow;
      b0 += 2 * g.btiles * g.bprow;
      g.cv0 = static_cast<int32_t>(c0);
      c0 += static_cast<int64_t>(g.btiles) * ((g.bgroups + kConvGroups - 1) / kConvGroups);
    }
    convs       = static_cast<int32_t>(c0);
    bconv_elems = std::max(bconv_elems, b0);
  };
  for (int32_t t = 0; t < S.nlevels; t++) {
    LevelPlan &L = levels[t];
    L.small_begin = static_cast<int32_t>(h_small.size());
    L.large_begin = static_cast<int32_t>(h_large.size());
    for (int64_t q = S.level_ptr[t]; q < S.level_ptr[t + 1]; q++) {
      const int32_t J = S.level_sup[q];
      (is_large(J) ? h_large : h_small).push_back(J);
    }
    L.small_count = static_cast<int32_t>(h_small.size()) - L.small_begin;
    L.large_count = static_cast<int32_t>(h_large.size()) - L.large_begin;
    // Extend-add: per phase (the parents' panel columns, then their update
    // matrices' columns) one CTA per chunk of kEaChunk parent columns that a
    // child adds to, with those children's hits in child order.
    std::vector<int32_t> task0(L.large_count);
    for (int32_t q = L.large_begin; q < L.large_begin + L.large_count; q++) {
      const int64_t P = h_large[q];
      task0[q - L.large_begin] = static_cast<int32_t>(tasks.size());
      for (int64_t c = S.child_ptr[P]; c < S.child_ptr[P + 1]; c++) {
        const int64_t C = S.child_list[c];
        EaTask        tk;
        tk.child_u = S.uofs[C];
        tk.rel     = S.srowptr[C] + S.w(C);
        tk.rc      = static_cast<int32_t>(S.h(C) - S.w(C));
        tk.pad     = 0;
        tasks.push_back(tk);
      }
    }
    for (int ph = 0; ph < 2; ph++) {
      L.ea_begin[ph] = static_cast<int32_t>(chunks_h.size());
      for (int32_t q = L.large_begin; q < L.large_begin + L.large_count; q++) {
        const int64_t P  = h_large[q];
        const int64_t nk = S.child_ptr[P + 1] - S.child_ptr[P];
        const int32_t hp = static_cast<int32_t>(S.h(P)), wp = static_cast<int32_t>(S.w(P));
        const int32_t lo = ph == 0 ? 0 : wp, hi = ph == 0 ? wp : hp;
        if (nk == 0 || hi <= lo) continue;
        const int32_t nch = (hi - lo + kEaChunk - 1) / kEaChunk;
        L.ea_rows[ph]     = std::max(L.ea_rows[ph], hp - lo);
        // Hits per chunk (counted, then placed), children in order: a child's
        // columns in one chunk are consecutive (its row map increases).
        std::vector<int32_t> cnt(nch + 1, 0);
        auto walk = [&](auto &&emit) {
          for (int64_t k = 0; k < nk; k++) {
            const int32_t  tix = task0[q - L.large_begin] + static_cast<int32_t>(k);
            const EaTask  &tk  = tasks[tix];
            const int32_t *rl  = S.srel.data() + tk.rel;
            int32_t        u   = 0;
            while (u < tk.rc && rl[u] < lo) u++;
            while (u < tk.rc && rl[u] < hi) {
              const int32_t ch = (rl[u] - lo) / kEaChunk, end = lo + (ch + 1) * kEaChunk;
              int32_t       v  = u;
              while (v < tk.rc && rl[v] < std::min(end, hi)) v++;
              emit(ch, tix, u, v);
              u = v;
            }
          }
        };
        walk([&](int32_t ch, int32_t, int32_t, int32_t) { cnt[ch + 1]++; });
        for (int32_t c = 0; c < nch; c++) cnt[c + 1] += cnt[c];
        const int32_t        hbase = static_cast<int32_t>(hits_h.size());
        std::vector<int32_t> fill(cnt.begin(), cnt.end() - 1);
        hits_h.resize(hits_h.size() + cnt[nch]);
        walk([&](int32_t ch, int32_t tix, int32_t u, int32_t v) {
          hits_h[hbase + fill[ch]++] = EaHit{tix, u, v, 0};
        });
        for (int32_t c = 0; c < nch; c++) {
          if (cnt[c + 1] == cnt[c]) continue;  // no child adds to these columns
          EaChunk ck;
          ck.parent_panel = S.slofs[P];
          ck.parent_u     = S.uofs[P];
          ck.hp           = hp;
          ck.wp           = wp;
          ck.c0           = lo + c * kEaChunk;
          ck.nc           = std::min(kEaChunk, hi - ck.c0);
          ck.hit0         = hbase + cnt[c];
          ck.hit1         = hbase + cnt[c + 1];
          chunks_h.push_back(ck);
        }
      }
      L.ea_count[ph] = static_cast<int32_t>(chunks_h.size()) - L.ea_begin[ph];
    }
    // Blocked steps.  Step kb: the left-looking update of block column kb
    // by the columns before it, then its diagonal block and panel solve;
    // after the last step the update matrix, in one product.
    int64_t maxw = 0;
    for (int32_t q = L.large_begin; q < L.large_begin + L.large_count; q++)
      maxw = std::max(maxw, S.w(h_large[q]));
    for (int64_t kb = 0; kb < maxw; kb += kNB) {
      LevelPlan::Step st{static_cast<int32_t>(descs.size()), 0, 0, 0,
                         static_cast<int32_t>(probs.size()), 0, 0, 0, 0};
      int64_t linv_top = 0;
      for (int32_t q = L.large_begin; q < L.large_begin + L.large_count; q++) {
        const int64_t J = h_large[q], w = S.w(J), h = S.h(J);
        if (w <= kb) continue;
        StepDesc d;
        d.panel  = S.slofs[J];
        d.uofs   = S.uofs[J];
        d.linv   = linv_top;
        d.h      = static_cast<int32_t>(h);
        d.w      = static_cast<int32_t>(w);
        d.kb     = static_cast<int32_t>(kb);
        d.nbk    = static_cast<int32_t>(std::min<int64_t>(kNB, w - kb));
        d.col0   = static_cast<int32_t>(S.sfirst[J]);
        const int64_t M = h - kb - d.nbk;
        d.trsm_tile0    = st.trsm_tiles;
        st.trsm_tiles += static_cast<int32_t>((M + kBM - 1) / kBM);
        d.upd_tile0       = 0;
        d.upd_panel_tiles = 0;
        trsm_flops += 2.0 * d.nbk * static_cast<double>(d.nbk) * static_cast<double>(M);
        if (kb > 0) {
          // Rows kb .. h-1 in the packed numbering: kb .. w-1, the gap up to
          // Wt, then the off-diagonal rows.
          const int64_t wt = pk_wt(J);
          GemmProb g{};
          g.a_ofs  = S.slofs[J] + kb;
          g.lda    = static_cast<int32_t>(h);
          g.c_ofs  = S.slofs[J] + kb + kb * h;
          g.ldc    = static_cast<int32_t>(h);
          g.d_ofs  = S.sfirst[J];
          g.prow   = pk_groups(J) * PackedFront::kGroupFloats;
          g.pa     = pk_ofs[J] + (kb / PackedFront::kRowTile) * g.prow;
          g.pb     = g.pa;
          g.pd     = pd_ofs[J];
          g.gap_at = static_cast<int32_t>(w - kb);
          g.gap    = static_cast<int32_t>(h > w ? wt - w : 0);
          g.M      = static_cast<int32_t>(h > w ? wt + (h - w) - kb : w - kb);
          g.N      = d.nbk;
          g.K      = static_cast<int32_t>(kb);
          g.c_in_u = 0;
          g.lower  = 1;
          probs.push_back(g);
        }
        d.pk           = pk_ofs[J];
        d.pd           = pd_ofs[J];
        d.pk_g         = static_cast<int32_t>(pk_groups(J));
        d.pk_wt        = static_cast<int32_t>(pk_wt(J));
        descs.push_back(d);
        st.count++;
        linv_top += (d.nbk + 31) / 32 * 32 * (int64_t)kNB;
        linv_elems = std::max(linv_elems, linv_top);
      }
      st.ll_count = static_cast<int32_t>(probs.size()) - st.ll_begin;
      finish_launch(st.ll_begin, st.ll_count, st.ll_tiles, st.ll_rtiles, st.ll_convs);
      L.steps.push_back(st);
    }
    L.u_begin = static_cast<int32_t>(probs.size());
    for (int32_t q = L.large_begin; q < L.large_begin + L.large_count; q++) {
      const int64_t J = h_large[q], w = S.w(J), h = S.h(J), r = h - w;
      if (r <= 0) continue;
      GemmProb g{};
      g.a_ofs  = S.slofs[J] + w;
      g.lda    = static_cast<int32_t>(h);
      g.c_ofs  = S.uofs[J];
      g.ldc    = static_cast<int32_t>(r);
      g.d_ofs  = S.sfirst[J];
      g.prow   = pk_groups(J) * PackedFront::kGroupFloats;
      g.pa     = pk_ofs[J] + (pk_wt(J) / PackedFront::kRowTile) * g.prow;
      g.pb     = g.pa;
      g.pd     = pd_ofs[J];
      g.gap_at = static_cast<int32_t>(r);
      g.gap    = 0;
      g.M = g.N = static_cast<int32_t>(r);
      g.K      = static_cast<int32_t>(w);
      g.c_in_u = 1;
      g.lower  = 1;
      probs.push_back(g);
    }
    L.u_count = static_cast<int32_t>(probs.size()) - L.u_begin;
    finish_launch(L.u_begin, L.u_count, L.u_tiles, L.u_rtiles, L.u_convs);
  }
  ndesc = static_cast<int64_t>(descs.size());
  panel_read_bytes = 0;
  for (int64_t J = 0; J < ns; J++) {
    const double w = static_cast<double>(S.w(J)), h = static_cast<double>(S.h(J));
    panel_read_bytes += 4.0 * (w * h - w * (w - 1) / 2);
  }
  // The host arrays stay with the plan, so an evicted plan can go back to
  // the device without being built again.
  host_.descs       = std::move(descs);
  host_.tasks       = std::move(tasks);
  host_.chunks      = std::move(chunks_h);
  host_.hits        = std::move(hits_h);
  host_.probs       = std::move(probs);
  build_flow();
  if (upload) upload_all(s);
}

size_t Plan::upload_bytes() const {
  auto b = [](const auto &v) { return v.size() * sizeof(v[0]); };
  return b(S.amap) + b(S.arow) + b(S.acol) + b(S.diag_pos) + b(S.Kp) + b(S.Kj) + b(S.Ksrc) +
         b(S.sfirst) + b(S.srowptr) + b(S.srows) + b(S.srel) + b(S.slofs) + b(S.uofs) +
         b(S.child_ptr) + b(S.child_list) + b(S.perm) + b(h_small) +
         b(host_.descs) + b(host_.tasks) + b(host_.chunks) + b(host_.hits) + b(host_.probs) +
         b(host_.flow_warp) + b(host_.flow_leaf) + b(host_.flow_fwd) + b(host_.flow_bwd) + b(host_.flow_inv) +
         b(host_.flow_gfirst) + b(host_.flow_gmore);
}

void Plan::upload_all(cudaStream_t s) {
  const auto t0 = std::chrono::steady_clock::now();
  amap       = upload(S.amap, s);
  arow       = upload(S.arow, s);
  acol       = upload(S.acol, s);
  diag_pos   = upload(S.diag_pos, s);
  Kp         = upload(S.Kp, s);
  Kj         = upload(S.Kj, s);
  Ksrc       = upload(S.Ksrc, s);
  sfirst     = upload(S.sfirst, s);
  srowptr    = upload(S.srowptr, s);
  srows      = upload(S.srows, s);
  srel       = upload(S.srel, s);
  slofs      = upload(S.slofs, s);
  uofs       = upload(S.uofs, s);
  child_ptr  = upload(S.child_ptr, s);
  child_list = upload(S.child_list, s);
  perm       = upload(S.perm, s);
  small_list = upload(h_small, s);
  steps      = upload(host_.descs, s);
  ea_tasks   = upload(host_.tasks, s);
  ea_chunks  = upload(host_.chunks, s);
  ea_hits    = upload(host_.hits, s);
  gemm_probs = upload(host_.probs, s);
  flow_warp    = upload(host_.flow_warp, s);
  flow_leaf    = upload(host_.flow_leaf, s);
  flow_fwd     = upload(host_.flow_fwd, s);
  flow_bwd     = upload(host_.flow_bwd, s);
  flow_inv     = upload(host_.flow_inv, s);
  flow_gfirst  = upload(host_.flow_gfirst, s);
  flow_gmore   = upload(host_.flow_gmore, s);
  MPIR_CUDA(cudaStreamSynchronize(s));
  upload_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  on_device = true;
}

void Plan::release_device() {
  for (DeviceBuffer *d :
       {&amap, &arow, &acol, &diag_pos, &Kp, &Kj, &Ksrc, &sfirst, &srowptr, &srows, &srel,
        &slofs, &uofs, &child_ptr, &child_list, &perm, &ea_chunks, &ea_hits, &small_list,
        &steps, &ea_tasks, &gemm_probs, &flow_warp, &flow_leaf, &flow_fwd,
        &flow_bwd, &flow_inv, &flow_gfirst, &flow_gmore})
    d->release();
  on_device = false;
}

void Numeric::allocate(const Plan &P) {
  release_graph();
  const Symbolic &S = P.S;
  panel.resize(std::max<int64_t>(S.panel_elems, 1) * sizeof(float));
  if (store_prec == 2 || store_prec == 3)
    panel16.resize(std::max<int64_t>(S.panel_elems, 1) * 2);
  else
    panel16.release();
  // Positions of the inverses that no column of a front has stay zero.
  wpanel.resize(std::max<int64_t>(P.flow_wpanel_total, 1) * sizeof(double));
  inv64.resize(std::max<int64_t>(P.flow_inv_elems, 1) * sizeof(double));
  device_zero(inv64.as<void>(), inv64.bytes());
  D.resize(std::max<int64_t>(S.n, 1) * sizeof(float));
  Dinv.resize(std::max<int64_t>(S.n, 1) * sizeof(float));
  status.resize(sizeof(FactorStatus));
  AD.resize(std::max<int64_t>(S.n, 1) * sizeof(double));
  Kval.resize(std::max<int64_t>(P.nnz_full, 1) * sizeof(double));
  Korig.resize(std::max<int64_t>(P.nnz_full, 1) * sizeof(double));
  has_scratch = false;
  ensure_scratch(P);
  valid = false;
}

void Numeric::ensure_scratch(const Plan &P) {
  if (has_scratch) return;
  release_graph();  // a recorded factorization points at the old buffers
  const Symbolic &S = P.S;
  if (!panel.bytes()) panel.resize(std::max<int64_t>(S.panel_elems, 1) * sizeof(float));
  uarena.resize(std::max<int64_t>(S.uarena_elems, 1) * sizeof(float));
  ws.resize(std::max<int64_t>(P.ws_elems, 1) * sizeof(float));
  // Packed fronts: positions that hold no value of L are never written and
  // stay zero from here on.
  bconv.resize(std::max<int64_t>(std::max(P.bconv_elems, P.linv_elems), 1) * sizeof(float));
  pack.resize(std::max<int64_t>(P.pk_elems, 1) * sizeof(float));
  packd.resize(std::max<int64_t>(2 * P.pd_elems, 1) * sizeof(float));
  device_zero(pack.as<void>(), pack.bytes());
  device_zero(packd.as<void>(), packd.bytes());
  Axs.resize(std::max<int64_t>(S.nnz, 1) * sizeof(double));
  Ax.resize(std::max<int64_t>(S.nnz, 1) * sizeof(double));
  has_scratch = true;
}

void Numeric::trim() {
  release_graph();
  for (DeviceBuffer *b : {&uarena, &ws, &bconv, &pack, &packd, &Axs, &Ax}) b->release();
  if (panel16.bytes()) panel.release();  // the solves read the 16-bit copy
  has_scratch = false;
}

size_t Numeric::bytes_for(const Plan &P, int store_prec) {
  const Symbolic &S  = P.S;
  auto            at = [](int64_t e, size_t b) { return std::max<int64_t>(e, 1) * b; };
  return at(S.panel_elems, store_prec == 1 ? 4 : 6) + at(S.uarena_elems, 4) +
         at(P.flow_inv_elems, 8) + at(P.flow_wpanel_total, 8) + at(P.ws_elems, 4) + at(std::max(P.bconv_elems, P.linv_elems), 4) +
         at(P.pk_elems, 4) + at(2 * P.pd_elems, 4) + 2 * at(S.n, 4) + sizeof(FactorStatus) +
         at(S.n, 8) + 2 * at(S.nnz, 8) + 2 * at(P.nnz_full, 8);
}

size_t Numeric::device_bytes() const {
  size_t b = 0;
  for (const DeviceBuffer *d : {&panel, &panel16, &uarena, &inv64, &wpanel, &D, &Dinv, &status,
                                &ws, &pack, &packd, &bconv, &AD, &Axs, &Kval, &Korig, &Ax})
    b += d->bytes();
  return b;
}

size_t Plan::device_bytes() const {
  size_t b = 0;
  for (const DeviceBuffer *d :
       {&amap, &arow, &acol, &diag_pos, &Kp, &Kj, &Ksrc, &sfirst, &srowptr, &srows, &srel,
        &slofs, &uofs, &child_ptr, &child_list, &perm, &ea_chunks, &ea_hits, &small_list,
        &steps, &ea_tasks, &gemm_probs, &flow_warp, &flow_leaf, &flow_fwd,
        &flow_bwd, &flow_inv, &flow_gfirst, &flow_gmore})
    b += d->bytes();
  return b;
}

static unsigned grid_for(int64_t n, int threads) {
  return static_cast<unsigned>((n + threads - 1) / threads);
}

__global__ void k_status_reset(FactorStatus *st) {
  if (threadIdx.x == 0) *st = FactorStatus{INT_MAX, 0, 0, 0};
}

void Numeric::release_graph() {
  if (graph) cudaGraphExecDestroy(graph);
  graph     = nullptr;
  ran_plain = false;
}

cudaGraph_t Numeric::record(const Plan &P, const double *d_Ax, double eps,
                            cudaStream_t capture_stream, int64_t *launches) {
  cudaGraph_t g = nullptr;
  MPIR_CUDA(cudaStreamSynchronize(capture_stream));
  MPIR_CUDA(cudaStreamBeginCapture(capture_stream, cudaStreamCaptureModeThreadLocal));
  LaunchCapture cap;
  try {
    run(P, d_Ax, eps, capture_stream);
  } catch (...) {
    cudaStreamEndCapture(capture_stream, &g);
    if (g) cudaGraphDestroy(g);
    throw;
  }
  MPIR_CUDA(cudaStreamEndCapture(capture_stream, &g));
  valid = false;  // recorded, not run
  if (launches) *launches = cap.count();
  return g;
}

void Numeric::run_graph(const Plan &P, const double *d_Ax, double eps, cudaStream_t s,
                        cudaStream_t capture_stream) {
  if (kernel_timer().enabled || P.S.n == 0) {  // per-class timing needs the plain launches
    run(P, d_Ax, eps, s);
    return;
  }
  const bool current = graph && graph_ax == d_Ax && graph_eps == eps && graph_mode == update_mode;
  // A factorization that may be the only one of these buffers (a new factor
  // of the serving engine, a drop-in Compute) runs its launches directly: a
  // recording pays the capture and the instantiation for a single replay.
  // The second one records the graph that every later one replays.
  if (!current && !ran_plain) {
    release_graph();
    run(P, d_Ax, eps, s);
    ran_plain = true;
    return;
  }
  if (!current) {
    release_graph();
    cudaGraph_t g = record(P, d_Ax, eps, capture_stream, &graph_launches);
    const cudaError_t e = cudaGraphInstantiate(&graph, g, 0);
    cudaGraphDestroy(g);
    MPIR_CUDA(e);
    graph_ax   = d_Ax;
    graph_eps  = eps;
    graph_mode = update_mode;
  }
  eps_uf = eps;
  MPIR_CUDA(cudaGraphLaunch(graph, s));
  launch_add(graph_launches);
  valid = true;
}

namespace {
// A branch of the graph that a stream is recording: what is launched between
// begin() and end() depends on what came before begin() only, and what follows
// join() on both.
class CaptureFork {
 public:
  explicit CaptureFork(cudaStream_t s) : s_(s) { capturing_ = query().first; }
  bool capturing() const { return capturing_; }
  bool forked() const { return !branch_.empty(); }
  void begin() { main_ = query().second; }
  void end() {
    branch_ = query().second;
    set(main_);
  }
  void join() {
    if (!forked()) return;
    std::vector<cudaGraphNode_t> all = query().second;
    for (cudaGraphNode_t b : branch_)
      if (std::find(all.begin(), all.end(), b) == all.end()) all.push_back(b);
    set(all);
  }

 private:
  std::pair<bool, std::vector<cudaGraphNode_t>> query() const {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    const cudaGraphNode_t  *deps   = nullptr;
    size_t                  n      = 0;
    MPIR_CUDA(cudaStreamGetCaptureInfo(s_, &status, nullptr, nullptr, &deps, &n));
    if (status != cudaStreamCaptureStatusActive) return {false, {}};
    return {true, std::vector<cudaGraphNode_t>(deps, deps + n)};
  }
  void set(std::vector<cudaGraphNode_t> deps) {
    MPIR_CUDA(cudaStreamUpdateCaptureDependencies(s_, deps.data(), deps.size(),
                                                  cudaStreamSetCaptureDependencies));
  }
  cudaStream_t                 s_;
  bool                         capturing_ = false;
  std::vector<cudaGraphNode_t> main_, branch_;
};
}  // namespace

void Numeric::run(const Plan &P, const double *d_Ax, double eps, cudaStream_t s) {
  if (!has_scratch) throw std::logic_error("factorization scratch released (ensure_scratch)");
  const Symbolic &S  = P.S;
  KernelTimer    &kt = kernel_timer();
  eps_uf             = eps;
  valid              = false;
  launch(k_status_reset, 1, 32, 0, s, status.as<FactorStatus>());
  MPIR_CUDA(cudaMemsetAsync(panel.as<void>(), 0, S.panel_elems * sizeof(float), s));
  if (S.n == 0) return;
  kt.begin(kKcScatter, s);
  launch(k_scaling, grid_for(S.n, 256), 256, 0, s, S.n, P.diag_pos.as<int64_t>(), d_Ax,
                                               eps, AD.as<double>());
  launch(k_scatter, grid_for(S.nnz, 256), 256, 0, s, 
      S.nnz, d_Ax, AD.as<double>(), P.arow.as<int32_t>(), P.acol.as<int32_t>(),
      P.amap.as<int64_t>(), Axs.as<double>(), panel.as<float>());
  launch(k_csr_values, grid_for(P.nnz_full, 256), 256, 0, s, 
      P.nnz_full, P.Ksrc.as<int64_t>(), Axs.as<double>(), d_Ax, Kval.as<double>(),
      Korig.as<double>());
  kt.end(s);
  MPIR_CHECK_LAUNCH();
  float        *pan = panel.as<float>(), *ua = uarena.as<float>();
  FactorStatus *st  = status.as<FactorStatus>();
  static const bool trsm_simt_env = [] {
    const char *e = std::getenv("MPIR_TRSM");
    return e != nullptr && std::string(e) == "simt";
  }();
  const bool trsm_tc = update_mode >= 0 && !trsm_simt_env;
  static OncePerDevice trsm_attr, diag_attr;
  const int            trsm_smem = kBM * (kBN + 1) * sizeof(float);
  const int            diag_smem = kDiagSmemFloats * sizeof(float);
  allow_smem(trsm_attr, trsm_smem, {reinterpret_cast<const void *>(k_step_gemm<true>)});
  allow_smem(diag_attr, diag_smem, {reinterpret_cast<const void *>(k_diag_block)});
  // Float64 inverses of the diagonal blocks for the triangular solves.  In a
  // recorded graph those below the last level form a branch of their own beside
  // it (its fronts are few and leave most of the chip idle; in a stream all of
  // them follow the last level).
  CaptureFork inverses(s);
  for (const LevelPlan &L : P.levels) {
    if (&L == &P.levels.back() && inverses.capturing()) {
      inverses.begin();
      flow_invert(P, *this, kFlowLow, s);
      inverses.end();
    }
    // Children's update matrices into the fronts' panels (the update
    // matrices' own columns follow after the product that defines them).
    auto extend_add = [&](int phase) {
      const int ph = phase - 1;
      if (L.ea_count[ph] > 0) {
        kt.begin(kKcExtendAdd, s);
        // Row parts: up to five CTAs an SM, at least 256 rows each.
        const int parts = std::clamp<int>(std::min(5 * kSMs / L.ea_count[ph], L.ea_rows[ph] / 256), 1, 16);
        launch(k_extend_add, dim3(L.ea_count[ph], parts), 256, 0, s,
               P.ea_chunks.as<EaChunk>() + L.ea_begin[ph],
               static_cast<const EaHit *>(P.ea_hits.as<EaHit>()),
               static_cast<const EaTask *>(P.ea_tasks.as<EaTask>()), P.srel.as<int32_t>(), pan,
               ua);
        kt.end(s);
      }
    };
    extend_add(1);
    if (L.small_count > 0) {
      kt.begin(kKcSmallFront, s);
      launch(k_small_fronts<kSmallFront>, L.small_count, kSmallThreads, 0, s, 
          P.small_list.as<int32_t>() + L.small_begin, P.sfirst.as<int64_t>(),
          P.srowptr.as<int64_t>(), P.slofs.as<int64_t>(), P.uofs.as<int64_t>(),
          P.child_ptr.as<int64_t>(), P.child_list.as<int32_t>(),
          P.srel.as<int32_t>(), pan, ua, D.as<float>(), Dinv.as<float>(), st);
      kt.end(s);
    }
    const GemmProb *gp = P.gemm_probs.as<GemmProb>();
    auto gemm = [&](int32_t begin, int32_t count, int32_t tiles, int32_t rtiles,
                    int32_t convs) {
      if (count <= 0 || tiles <= 0) return;
      kt.begin(kKcUpdate, s);
      if (update_mode == 1 && convs > 0)
        launch_convert_b(gp + begin, count, convs, pack.as<float>(), packd.as<float>(),
                         bconv.as<float>(), s);
      if (update_mode < 0)
        launch(k_gemm_simt, tiles, kGemmThreads, 0, s, gp + begin, count, pan, ua,
               static_cast<const float *>(D.as<float>()), ws.as<float>());
      else
        launch_gemm_tc(update_mode, gp + begin, count, tiles, pack.as<float>(),
                       packd.as<float>(), packd.as<float>() + P.pd_elems, bconv.as<float>(),
                       pan, ua, ws.as<float>(), st, s);
      kt.end(s);
      if (rtiles > 0) {
        kt.begin(kKcReduce, s);
        launch(k_split_reduce, rtiles * kReduceSlices, 256, 0, s, gp + begin, count,
               pan, ua, static_cast<const float *>(ws.as<float>()));
        kt.end(s);
      }
    };
    for (const auto &stp : L.steps) {
      const StepDesc *dd = P.steps.as<StepDesc>() + stp.begin;
      gemm(stp.ll_begin, stp.ll_count, stp.ll_tiles, stp.ll_rtiles, stp.ll_convs);
      kt.begin(kKcDiag, s);
      launch(k_diag_block, stp.count, kDiagThreads, diag_smem, s, dd, pan, bconv.as<float>(),
             D.as<float>(), Dinv.as<float>(), packd.as<float>(),
             packd.as<float>() + P.pd_elems, st);
      kt.end(s);
      if (stp.trsm_tiles > 0) {
        kt.begin(kKcTrsm, s);
        if (trsm_tc)
          launch_trsm_tc(dd, stp.count, stp.trsm_tiles, pan, bconv.as<float>(), Dinv.as<float>(),
                         pack.as<float>(), st, s);
        else
          launch(k_step_gemm<true>, stp.trsm_tiles, kGemmThreads, trsm_smem, s, dd, stp.count,
                 pan, ua, bconv.as<float>(), Dinv.as<float>(), pack.as<float>());
        kt.end(s);
      }
    }
    gemm(L.u_begin, L.u_count, L.u_tiles, L.u_rtiles, L.u_convs);
    extend_add(2);
    MPIR_CHECK_LAUNCH();
  }
  kt.begin(kKcDiag, s);
  flow_invert(P, *this, inverses.forked() ? kFlowTop : kFlowAll, s);
  inverses.join();
  kt.end(s);
  if (panel16.bytes() && S.panel_elems) {
    kt.begin(kKcScatter, s);
    launch(k_panel_to16, static_cast<unsigned>(std::min<int64_t>((S.panel_elems + 255) / 256, 148 * 16)),
           256, 0, s, S.panel_elems, panel.as<float>(), panel16.as<uint16_t>(),
           store_prec == 2 ? 1 : 0);
    kt.end(s);
  }
  valid = true;
}

int64_t Numeric::result(cudaStream_t s, int32_t *zero_col, bool *nonfinite) const {
  FactorStatus h;
  MPIR_CUDA(cudaMemcpyAsync(&h, status.as<void>(), sizeof h, cudaMemcpyDeviceToHost, s));
  MPIR_CUDA(cudaStreamSynchronize(s));
  if (zero_col) *zero_col = h.zero_pivot;
  if (nonfinite) *nonfinite = h.nonfinite != 0;
  if (h.timeout) return -5;
  if (h.zero_pivot != INT_MAX) return -1;
  return h.npos;
}

// ---------------------------------------------------------------------------
namespace {
std::atomic<int64_t>        g_launches{0};
thread_local LaunchCapture *t_capture = nullptr;
}  // namespace

int64_t launch_total() { return g_launches.load(std::memory_order_relaxed); }

void launch_add(int64_t n) {
  if (t_capture)
    t_capture->add(n);
  else
    g_launches.fetch_add(n, std::memory_order_relaxed);
}

LaunchCapture::LaunchCapture() : outer_(t_capture) { t_capture = this; }
LaunchCapture::~LaunchCapture() { t_capture = outer_; }

KernelTimer &kernel_timer() {
  static KernelTimer t;
  return t;
}

void KernelTimer::begin(int c, cudaStream_t s) {
  if (!enabled) return;
  cudaEvent_t a, b;
  cudaEventCreate(&a);
  cudaEventCreate(&b);
  cudaEventRecord(a, s);
  ev.push_back(a);
  ev.push_back(b);
  cls.push_back(c);
}

void KernelTimer::end(cudaStream_t s) {
  if (!enabled) return;
  cudaEventRecord(ev.back(), s);
}

void KernelTimer::reset() {
  for (auto e : ev) cudaEventDestroy(e);
  ev.clear();
  cls.clear();
}

void KernelTimer::collect(double *ms, int64_t *count, int nclass) {
  for (int c = 0; c < nclass; c++) {
    ms[c]    = 0;
    count[c] = 0;
  }
  for (size_t i = 0; i < cls.size(); i++) {
    float t = 0;
    cudaEventElapsedTime(&t, ev[2 * i], ev[2 * i + 1]);
    if (cls[i] < nclass) {
      ms[cls[i]] += t;
      count[cls[i]] += 1;
    }
  }
}

}  // namespace mpir
