// Triangular solves with the supernodal LDL^T factor on the GPU.
//
// Computes x <- L^{-T} D^{-1} L^{-1} x, the preconditioner application that
// QDLDL_solve performs column by column (qdldl.hpp:362-432), over the
// supernodal elimination tree:
//   forward   each front takes its own right-hand side entries plus its
//             children's update vectors, solves with its unit-lower diagonal
//             block and leaves L_{R,J} x_J (negated, accumulated) as its own
//             update vector for its parent;
//   diagonal  x <- Dinv .* x, read by the backward solve;
//   backward  each front gathers the finished x of its row set R_J and solves
//             with L_J^T.
// Each direction is one launch for the whole tree.  CTAs take work items by
// ticket in an order in which an item waits only on earlier ones (leaves to
// root, or root to leaves), and every value that passes between items (an
// update vector entry, a block result, a partial sum) is its own ready
// signal: it is stored once over a pending marker, and the items that need it
// poll it (solve_dev.cuh).  No level waits for another as a whole: what bounds
// a direction is the chain of hand-overs from the leaves to the root (about
// three per level, 1 to 1.5 us each) and, inside the root, two per 512
// columns, or the bytes of L where they are many.
//
// Diagonal blocks are applied through their inverse, computed in float64
// from the float32 factor per super-block of 512 columns (k_flow_invert).
// Per 128 columns, as before, the n = 40,960 system's root (9,317 columns)
// was a chain of 73 block products; per 512 it is 19, each spread over 16
// CTAs.  A wider block would shorten the chain further, but its share per
// CTA of 32 rows no longer fits in shared memory.
//
// Measured, one application (forward + backward, float32 factor), against the
// solves by levels of 128-row blocks that this replaced (events around each
// launch, both on one box): n = 1,280: 0.079 ms (0.183); n = 2,160: 0.088 (0.249);
// n = 24,603: 0.26 (0.74); n = 40,960: 0.41 (0.98), 283 MB of L read twice at 1.4
// TB/s; n = 138,240: 2.1 (3.1), 2.6 GB read twice at 2.5 TB/s.
// Vectors are float64, the factor float32 or 16-bit (widened on load), as
// QDLDL_solve with FACTPREC = float and XPREC = double.  Sums have a fixed
// order, so results do not depend on scheduling.
#include <algorithm>
#include <atomic>
#include <string>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "engine.hpp"
#include "solve.hpp"
#include "solve_dev.cuh"
#include "flow_dev.cuh"

namespace mpir {

// Shared memory (doubles): kFlowInvSmem, written by bulk copies only, then 4,608
// for vectors and partial sums.
constexpr int kFlowSmem      = kFlowInvSmem + 4608;
constexpr int kFlowSmemBytes = kFlowSmem * sizeof(double);

__global__ void k_mark_pending(int64_t n, double *p) {
  flow_mark(p, n);
}

void flow_pending(double *p, int64_t n, cudaStream_t s) {
  launch(k_mark_pending, static_cast<unsigned>(std::min<int64_t>((n + 255) / 256, kSMs * 16)), 256, 0, s,
         n, p);
}

// sum_k l[k] y[k] over 32 entries of shared memory (16-byte aligned).
template <class V>
__device__ __forceinline__ double dot32(const V (&l)[32], const double *y) {
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    const double2 a = *reinterpret_cast<const double2 *>(y + k);
    const double2 b = *reinterpret_cast<const double2 *>(y + k + 2);
    s0 += static_cast<double>(l[k]) * a.x;
    s1 += static_cast<double>(l[k + 1]) * a.y;
    s2 += static_cast<double>(l[k + 2]) * b.x;
    s3 += static_cast<double>(l[k + 3]) * b.y;
  }
  return (s0 + s1) + (s2 + s3);
}

// sum_k m[P k] y[k] over 32 entries, both in shared memory.
template <int P>
__device__ __forceinline__ double dot_pitch(const double *m, const double *y) {
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    const double2 a = *reinterpret_cast<const double2 *>(y + k);
    const double2 b = *reinterpret_cast<const double2 *>(y + k + 2);
    s0 += m[P * k] * a.x;
    s1 += m[P * (k + 1)] * a.y;
    s2 += m[P * (k + 2)] * b.x;
    s3 += m[P * (k + 3)] * b.y;
  }
  return (s0 + s1) + (s2 + s3);
}

// ---------------------------------------------------------------------------
// Forward.

// sum_c L(r, c) y_c over the columns c < cend of a wide front, tile by tile
// (512 / RG columns) as the block results y become ready: warp v takes the
// rows 32 (v % RG) .. (lane) and the columns 32 (v / RG) .. of each tile;
// the next tile's L values are loaded while the current one waits, so that a
// CTA that starts late catches up at two tiles in flight.  The last tile (the
// result just before on the chain) is widened before its wait: conversions
// run at a quarter of the FMA rate and would be on the chain.
template <int RG, class T>
__device__ __forceinline__ double rows_apply(const FlowArgs<T> &a, const T *P, int64_t h, int64_t r,
                                             bool rok, int cend, const double *y, double *yw,
                                             long polls) {
  constexpr int TW = 512 / RG;
  const int     warp = threadIdx.x / 32, lane = threadIdx.x % 32, cq = 32 * (warp / RG);
  const int     tiles = (cend + TW - 1) / TW;
  if (tiles == 0) return 0.0;
  double  acc = 0.0;
  double *yv  = yw + 32 * warp;
  float   lv[32], lvn[32];
  auto    load_y = [&](int c) { return c + lane < cend ? ld_relaxed_u64(y + c + lane) : 0ull; };
  load_cols(lv, P, h, r, rok, cq, cend);
  unsigned long long raw = load_y(cq);
  for (int b = 0; b + 1 < tiles; b++) {
    const int c = b * TW + cq;
    load_cols(lvn, P, h, r, rok, c + TW, cend);
    const unsigned long long rawn = b + 2 < tiles ? load_y(c + TW) : 0ull;
    yv[lane] = c + lane < cend ? take_value(raw, y + c + lane, a.err, polls) : 0.0;
    __syncwarp();
    acc += dot32(lv, yv);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 32; k++) lv[k] = lvn[k];
    raw = rawn;
  }
  const int c = (tiles - 1) * TW + cq;
  double    ld[32];
#pragma unroll
  for (int k = 0; k < 32; k++) ld[k] = static_cast<double>(lv[k]);
  yv[lane] = c + lane < cend ? wait_value(y + c + lane, a.err, polls) : 0.0;
  __syncwarp();
  acc += dot32(ld, yv);
  return acc;
}

// kFwdNarrow (w <= 128): y_J = Inv z_J, then up to 512 of the rows below,
// u = z_R - L_{R,J} y_J.  Every item of the front computes y_J itself (w
// values), which saves a hand-over; the first one keeps it.  RG = 16 (w <= 32):
// a thread a row; RG = 4: tiles of 128 rows, a quarter of the columns each
// (the next tile's L values are loaded while the current one is applied).
// Thread tid gathers and stores row tid of the item.
template <int RG, class T>
__device__ __noinline__ void fwd_narrow(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I, FlowSlot &N,
                                        double *sm, uint32_t &phase) {
  const FlowFront &f   = I.item.f;
  const int        tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int        w = f.w, nbw = (w + 31) / 32, nr = I.item.nr;
  const long       polls = I.polls;
  double          *inv = sm, *zs = sm + kFlowInvSmem, *ys = zs + 512, *part = ys + 512;
  const uint32_t   bar = smem_addr(&S.bar);
  if (tid == 0) {
    const uint32_t bytes = nbw * (nbw + 1) / 2 * kFlowBlk * sizeof(double);
    bulk_expect(bar, bytes);
    bulk_get(inv, a.inv + f.inv, bytes, bar);
  }
  constexpr int kTile = 32 * RG;
  const int     cq = warp / RG, rt = tid % kTile;
  const int64_t r0 = I.item.r0;
  const T      *P  = a.panel + f.panel;
  float         lv[32], lvn[32];
  load_cols(lv, P, f.h, r0 + rt, rt < nr, 32 * cq, w);
  flow_fetch(a, N);
  Gather<1> gz, gr;
  if (tid < w) gz.begin(a, f.zofs + tid, a.z);
  if (tid < nr) gr.begin(a, f.zofs + r0 + tid, a.z);
  if (tid < 32 * nbw) zs[tid] = tid < w ? gz.finish(a, a.z, a.x[f.col0 + tid], polls) : 0.0;
  __syncthreads();
  bulk_wait(bar, phase, a.err);
  phase ^= 1;
  const int bi = warp / 4, bj = warp % 4;
  if (bi < nbw && bj <= bi) {
    const double *blk = inv + (bi * (bi + 1) / 2 + bj) * kFlowBlk + lane;
    double        iv[32];
#pragma unroll
    for (int c = 0; c < 32; c++) iv[c] = blk[33 * c];
    part[bj * 128 + 32 * bi + lane] = dot32(iv, zs + 32 * bj);
  }
  __syncthreads();
  if (tid < 128) {
    double y = 0.0;
    if (tid < w)
      for (int j = 0; j <= tid / 32; j++) y += part[j * 128 + tid];
    ys[tid] = y;
    if (tid < w && r0 == w) a.f[f.col0 + tid] = y;
  }
  __syncthreads();
  double acc = 0.0;
  if (RG == 16) {
    acc = dot32(lv, ys);
  } else {
    for (int q = 0; q * kTile < nr; q++) {
      const int rn = (q + 1) * kTile + rt;
      if ((q + 1) * kTile < nr) load_cols(lvn, P, f.h, r0 + rn, rn < nr, 32 * cq, w);
      part[(4 * q + cq) * 128 + rt] = dot32(lv, ys + 32 * cq);
#pragma unroll
      for (int k = 0; k < 32; k++) lv[k] = lvn[k];
    }
    __syncthreads();
    const double *p = part + tid / 128 * 512 + tid % 128;
    if (tid < nr) acc = (p[0] + p[128]) + (p[256] + p[384]);
  }
  if (tid < nr) {
    const double u = gr.finish(a, a.z, 0.0, polls) - acc;
    if (I.publish) st_relaxed_f64(a.z + f.zofs + r0 + tid, u);
  }
}

// kFwdSlab (w > 128): 32 rows of the diagonal block.  z = its right-hand side
// less the columns of the super-blocks before its own, handed to the other
// slabs of the super-block; then y = the slab's rows of the inverse times
// their z: warp 0 takes the diagonal 32 x 32 block, warp v the block v - 1.
template <class T>
__device__ __noinline__ void fwd_slab(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I, FlowSlot &N,
                                      double *sm, uint32_t &phase) {
  const FlowFront &f   = I.item.f;
  const int        tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const long       polls = I.polls;
  const int        r0 = I.item.r0, s = r0 / kFlowSB, i = (r0 % kFlowSB) / 32;
  const bool       rok = lane < I.item.nr, last = r0 + 32 >= f.w || i == 15;
  double          *inv = sm, *yw = sm + kFlowInvSmem, *part = yw + 512, *part2 = part + 512;
  const uint32_t   bar = smem_addr(&S.bar);
  if (tid == 0) {
    const uint32_t bytes = (i + 1) * kFlowBlk * sizeof(double);
    bulk_expect(bar, bytes);
    bulk_get(inv, a.inv + f.inv + (static_cast<int64_t>(s) * kFlowTriSB + i * (i + 1) / 2) * kFlowBlk,
             bytes, bar);
  }
  flow_fetch(a, N);
  double zr = 0.0;
  if (warp == 0 && rok) {
    Gather<1> g;
    g.begin(a, f.zofs + r0 + lane, a.z);
    zr = g.finish(a, a.z, a.x[f.col0 + r0 + lane], polls);
  }
  const double *y = a.y + (I.ticket % kFlowCopies) * a.n + f.col0;
  if (s > 0) {
    part[32 * warp + lane] = rows_apply<1>(a, a.panel + f.panel, f.h, r0 + lane, rok,
                                           s * kFlowSB, y, yw, polls);
    __syncthreads();
  }
  double *yz = a.yz + f.col0 + s * kFlowSB;
  if (warp == 0) {
    if (s > 0) {
      double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int v = 0; v < 16; v++) t[v % 4] += part[32 * v + lane];
      zr -= (t[0] + t[1]) + (t[2] + t[3]);
    }
    if (!last && I.publish) st_relaxed_f64(yz + 32 * i + lane, zr);
  }
  bulk_wait(bar, phase, a.err);
  phase ^= 1;
  if (warp <= i) {
    const int     j   = warp == 0 ? i : warp - 1;
    const double *blk = inv + j * kFlowBlk + lane;
    double        iv[32];
#pragma unroll
    for (int c = 0; c < 32; c++) iv[c] = blk[33 * c];
    if (warp > 0) zr = wait_value(yz + 32 * j + lane, a.err, polls);
    yw[32 * warp + lane] = zr;
    __syncwarp();
    part2[32 * warp + lane] = dot32(iv, yw + 32 * warp);
  }
  __syncthreads();
  if (warp == 0 && rok) {
    double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int v = 0; v < 16; v++)
      if (v <= i) t[v % 4] += part2[32 * v + lane];
    const double  yv = (t[0] + t[1]) + (t[2] + t[3]);
    const int64_t g  = f.col0 + r0 + lane;
    if (I.publish) {
#pragma unroll
      for (int c = 0; c < kFlowCopies; c++) st_relaxed_f64(a.y + c * a.n + g, yv);
    }
    a.f[g] = yv;
  }
}

// kFwdRows (w > 128): 128 rows below the diagonal block.
template <class T>
__device__ __noinline__ void fwd_rows(const FlowArgs<T> &a, const FlowSlot &I, FlowSlot &N,
                                       double *sm) {
  const FlowFront &f   = I.item.f;
  const int        tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const long       polls = I.polls;
  double          *yw = sm + kFlowInvSmem, *part = yw + 512;
  const int64_t    r   = I.item.r0 + 32 * (warp % 4) + lane;
  const bool       rok = r < I.item.r0 + I.item.nr;
  Gather<1>        g;
  if (rok && warp < 4) g.begin(a, f.zofs + r, a.z);
  flow_fetch(a, N);
  const double *y = a.y + (I.ticket % kFlowCopies) * a.n + f.col0;
  part[(warp / 4) * 128 + tid % 128] =
      rows_apply<4>(a, a.panel + f.panel, f.h, r, rok, f.w, y, yw, polls);
  __syncthreads();
  if (rok && warp < 4) {
    const double *p = part + tid;
    const double  u = g.finish(a, a.z, 0.0, polls) - ((p[0] + p[128]) + (p[256] + p[384]));
    if (I.publish) st_relaxed_f64(a.z + f.zofs + r, u);
  }
}

// z -= M(:, k) y_k over the columns, for the first 32 RT rows (those at or past
// h read what lies behind the panel and are not used).  No branch inside the
// loop: one warp alone hides latency only by what a column has in flight.
template <int RT>
__device__ __forceinline__ void warp_columns(const double *M, int ld, int w, const double *y,
                                             double (&z)[8]) {
#pragma unroll 4
  for (int k = 0; k < w; k++) {
    const double yk = y[k];
#pragma unroll
    for (int t = 0; t < RT; t++) z[t] -= M[k * ld + 32 * t] * yk;
  }
}

// kFwdSum: 16 lanes a sum, two contributions a lane.  A thread alone, as for the
// rows with few, took 2.2 ms for the 13,000 contributions of a star's centre, longer
// than the levels' solves before (1.0 ms an application; 5.4 so).
template <class T>
__device__ __noinline__ void fwd_sum(const FlowArgs<T> &a, const FlowSlot &I, FlowSlot &N) {
  const int tid = threadIdx.x, e = tid / 16, l = tid % 16;
  uint32_t  ix[2] = {kFlowNone, kFlowNone};
  if (e < I.item.nr) {
    const uint32_t *m = a.gmore + I.item.f.rows + kFlowFan * e + 2 * l;
    ix[0]             = m[0];
    ix[1]             = m[1];
  }
  flow_fetch(a, N);
  double z[2] = {0.0, 0.0};
  add_values<2>(a.z, ix, z, a.err, I.polls);
  double s = z[0] + z[1];
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (l == 0 && e < I.item.nr && I.publish) st_relaxed_f64(a.z + I.item.f.zofs + e, s);
}

// kFlowWarps: one front of w <= 32, h <= 256 per warp; lane l holds rows
// l + 32 t.  The rows' child contributions are polled together, one of each
// row at a time; then y = Inv z, and the rows below less L y.
template <class T>
__device__ __noinline__ void fwd_warp(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I, FlowSlot &N,
                                      double *sm, uint32_t &wphase) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (warp >= I.item.nr) {
    flow_fetch(a, N);
    return;
  }
  const long      polls = I.polls;
  const FlowFront f = a.warps[I.item.r0 + warp];
  const int       w = f.w, h = f.h, ld = h | 1;
  const uint32_t  bar = smem_addr(&S.wbar[warp]);
  const double   *M   = warp_panel(a, f, sm, bar) + lane;
  double         *zs  = sm + kFlowInvSmem + 64 * warp, *ys = zs + 32;
  constexpr int   RT = kWarpSolveH / 32;
  uint32_t        ix[RT], more[RT];
  double          z[RT];
#pragma unroll
  for (int t = 0; t < RT; t++) {
    FlowGather g = {kFlowNone, kFlowNone};
    if (lane + 32 * t < h) g = a.gfirst[f.zofs + lane + 32 * t];
    ix[t]   = g.first;
    more[t] = g.more;
    z[t]    = 0.0;
  }
  if (lane < w) z[0] = a.x[f.col0 + lane];
  flow_fetch(a, N);
  add_values<RT>(a.z, ix, z, a.err, polls);
  // the rows with further children: their lists, one entry of each at a time
  uint32_t n[RT];
  bool     any = false;
#pragma unroll
  for (int t = 0; t < RT; t++) {
    n[t] = more[t] != kFlowNone ? a.gmore[more[t]] : 0;
    any |= n[t] > 0;
  }
  for (uint32_t q = 0; __any_sync(0xffffffffu, any); q++) {
    any = false;
#pragma unroll
    for (int t = 0; t < RT; t++) {
      ix[t] = q < n[t] ? a.gmore[static_cast<int64_t>(more[t]) + 1 + q] : kFlowNone;
      any |= q + 1 < n[t];
    }
    add_values<RT>(a.z, ix, z, a.err, polls);
  }
  zs[lane] = z[0];
  __syncwarp();
  bulk_wait(bar, wphase, a.err);
  wphase ^= 1;
  double y0 = 0.0, y1 = 0.0;
  int    k  = 0;
#pragma unroll 4
  for (; k + 1 < w; k += 2) {
    y0 += M[k * ld] * zs[k];
    y1 += M[(k + 1) * ld] * zs[k + 1];
  }
  if (k < w) y0 += M[k * ld] * zs[k];
  ys[lane] = y0 + y1;  // entries at or past w are not used
  __syncwarp();
  if (h <= 64)
    warp_columns<2>(M, ld, w, ys, z);
  else if (h <= 128)
    warp_columns<4>(M, ld, w, ys, z);
  else
    warp_columns<8>(M, ld, w, ys, z);
  if (lane < w) a.f[f.col0 + lane] = y0 + y1;
#pragma unroll
  for (int t = 0; t < RT; t++) {
    const int i = lane + 32 * t;
    if (i >= w && i < h && I.publish) st_relaxed_f64(a.z + f.zofs + i, z[t]);
  }
}

// SUMS: of a plan with kFwdSum items (the others' kernel took 0.5 us longer with their
// case in it).
template <class T, bool SUMS>
__global__ void __launch_bounds__(kFlowThreads, 1) k_fwd_flow(const __grid_constant__ FlowArgs<T> a) {
  grid_wait();
  extern __shared__ __align__(128) double sm[];
  __shared__ __align__(16) FlowShared S;
  uint32_t phase = 0, wphase = 0;
  if (flow_idle(a)) return;
  flow_loop<false>(a, S, [&](const FlowSlot &I, FlowSlot &N) {
    switch (I.item.kind) {
      case kFlowWarps: fwd_warp(a, S, I, N, sm, wphase); break;
      case kFwdNarrow:
        if (I.item.f.w <= 32)
          fwd_narrow<16>(a, S, I, N, sm, phase);
        else
          fwd_narrow<4>(a, S, I, N, sm, phase);
        break;
      case kFwdSlab: fwd_slab(a, S, I, N, sm, phase); break;
      default:
        if (SUMS && I.item.kind == kFwdSum)
          fwd_sum(a, I, N);
        else
          fwd_rows(a, I, N, sm);
    }
  });
  flow_mark(a.mark, a.nmark);
}

// ---------------------------------------------------------------------------
// Backward.

// Sums of the warp's two columns over its lanes: the lower half of the warp
// ends with column 0, the upper half with column 1.
__device__ __forceinline__ double sum2(double s0, double s1) {
  const bool up = threadIdx.x & 16;
  double     s  = (up ? s1 : s0) + __shfl_xor_sync(0xffffffffu, up ? s0 : s1, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// The x values of the front's rows w + 512 c .. (nr of them) into xs.
template <class T>
__device__ __forceinline__ void get_rows(const FlowArgs<T> &a, const FlowFront &f, int64_t rb, int nr,
                                         double *xs, long polls) {
  const int tid = threadIdx.x;
  const int row = tid < nr ? a.srows[f.rows + rb + tid] : -1;
  wait_gate(a, f.gate, polls);
  xs[tid] = row >= 0 ? wait_value(a.xr + row, a.err, polls) : 0.0;
  __syncthreads();
}

// t_c = sum_r L(r, c) x_r over up to 512 rows below the block, for columns
// [c0, cend): emit(c, t_c) by one lane a column.
template <class T, class Emit>
__device__ __forceinline__ void chunk_cols(const FlowArgs<T> &a, const FlowFront &f, int64_t rb,
                                           int nr, int c0, int cend, double *xs, long polls,
                                           FlowSlot &N, Emit emit) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const T  *P = a.panel + f.panel;
  float     lv[2][16], lvn[2][16];
  load_rows(lv, P, f.h, rb, nr, c0, cend);
  flow_fetch(a, N);
  // The first tile is widened before the wait (see rows_apply).
  double ld[2][16];
#pragma unroll
  for (int j = 0; j < 2; j++)
#pragma unroll
    for (int i = 0; i < 16; i++) ld[j][i] = static_cast<double>(lv[j][i]);
  if (c0 + 32 < cend) load_rows(lv, P, f.h, rb, nr, c0 + 32, cend);
  get_rows(a, f, rb, nr, xs, polls);
  const int dc = 2 * warp + (lane >> 4);  // the lane's column of a tile
  {
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const double xv = xs[lane + 32 * i];
      s0 += ld[0][i] * xv;
      s1 += ld[1][i] * xv;
    }
    const double t = sum2(s0, s1);
    if ((lane & 15) == 0 && c0 + dc < cend) emit(c0 + dc, t);
  }
  for (int c = c0 + 32; c < cend; c += 32) {
    if (c + 32 < cend) load_rows(lvn, P, f.h, rb, nr, c + 32, cend);
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const double xv = xs[lane + 32 * i];
      s0 += static_cast<double>(lv[0][i]) * xv;
      s1 += static_cast<double>(lv[1][i]) * xv;
    }
    const double t = sum2(s0, s1);
    if ((lane & 15) == 0 && c + dc < cend) emit(c + dc, t);
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int i = 0; i < 16; i++) lv[j][i] = lvn[j][i];
  }
}

template <class T>
__device__ __noinline__ void bwd_chunk(const FlowArgs<T> &a, const FlowSlot &I, FlowSlot &N,
                                       double *sm) {
  const FlowFront &f  = I.item.f;
  const int        c  = I.item.c0;
  const int64_t    rb = f.w + static_cast<int64_t>(c) * kFlowChunk;
  const int        nr = static_cast<int>(min(static_cast<int64_t>(kFlowChunk), f.h - rb));
  double          *pp = a.part + f.part + static_cast<int64_t>(c) * f.w;
  chunk_cols(a, f, rb, nr, I.item.r0, I.item.r0 + I.item.nr, sm + kFlowInvSmem,
             I.polls, N, [&](int col, double t) { st_relaxed_f64(pp + col, t); });
}

// kBwdNarrow (w <= 128): x_J = Inv^T (z_J - t), t the rows below: the chunk
// partials, or (at most 512 rows) computed here.
template <class T>
__device__ __noinline__ void bwd_narrow(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I, FlowSlot &N,
                                        double *sm, uint32_t &phase) {
  const FlowFront &f   = I.item.f;
  const int        tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int        w = f.w, nbw = (w + 31) / 32;
  const long       polls = I.polls;
  double          *inv = sm, *xs = sm + kFlowInvSmem, *vs = xs + 512, *red = vs + 512,
                  *part = red + 512;
  const uint32_t   bar = smem_addr(&S.bar);
  if (tid == 0) {
    const uint32_t bytes = nbw * (nbw + 1) / 2 * kFlowBlk * sizeof(double);
    bulk_expect(bar, bytes);
    bulk_get(inv, a.inv + f.inv, bytes, bar);
  }
  double v = 0.0;
  if (tid < w) {
    v = a.f[f.col0 + tid];
    if (a.Dinv) v *= static_cast<double>(a.Dinv[f.col0 + tid]);
  }
  red[tid] = 0.0;
  if (f.chunks > 0 || f.h == w) flow_fetch(a, N);
  if (f.chunks > 0) {
    const int k = tid % 128, q = tid / 128;
    double    s = 0.0;
    if (k < w)
      for (int c = q; c < f.chunks; c += 4)
        s += wait_value(a.part + f.part + static_cast<int64_t>(c) * w + k, a.err, polls);
    red[tid] = s;
  } else if (f.h > w) {
    __syncthreads();
    chunk_cols(a, f, w, f.h - w, 0, w, xs, polls, N, [&](int col, double t) { red[col] = t; });
  }
  __syncthreads();
  if (tid < 128) vs[tid] = v - ((red[tid] + red[tid + 128]) + (red[tid + 256] + red[tid + 384]));
  __syncthreads();
  bulk_wait(bar, phase, a.err);
  phase ^= 1;
  const int bj = warp % 4, bi = warp / 4;
  if (bi < nbw && bj <= bi) {
    const double *blk = inv + (bi * (bi + 1) / 2 + bj) * kFlowBlk + 33 * lane;
    part[bi * 128 + 32 * bj + lane] = dot_pitch<1>(blk, vs + 32 * bi);
  }
  __syncthreads();
  if (tid < w) {
    double xo = 0.0;
    for (int i = tid / 32; i < nbw; i++) xo += part[i * 128 + tid];
    st_relaxed_f64(a.xr + f.col0 + tid, xo);
    a.x[f.col0 + tid] = xo;
  }
}

// kBwdSlab (w > 128): 32 columns of the diagonal block, the mirror of
// fwd_slab: t = the chunk partials + the rows of the super-blocks after its
// own, last first; v = z - t handed to the slabs before it in the
// super-block; x = the slab's columns of the inverse times v.
template <class T>
__device__ __noinline__ void bwd_slab(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I, FlowSlot &N,
                                      double *sm, uint32_t &phase) {
  const FlowFront &f   = I.item.f;
  const int        tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const long       polls = I.polls;
  const int        w = f.w, k0 = I.item.r0, s = k0 / kFlowSB, j = (k0 % kFlowSB) / 32;
  const int        nsl = min(16, (w - s * kFlowSB + 31) / 32), nsb = (w + kFlowSB - 1) / kFlowSB;
  const bool       ok = lane < I.item.nr;
  double          *inv = sm, *xs = sm + kFlowInvSmem, *part = xs + 1024, *ts = part + 512;
  __shared__ double ts2[32];
  const uint32_t   bar = smem_addr(&S.bar);
  if (tid == 0) {
    bulk_expect(bar, (nsl - j) * kFlowBlk * sizeof(double));
    for (int i = j; i < nsl; i++)
      bulk_get(inv + (i - j) * kFlowBlk,
               a.inv + f.inv +
                   (static_cast<int64_t>(s) * kFlowTriSB + i * (i + 1) / 2 + j) * kFlowBlk,
               kFlowBlk * sizeof(double), bar);
  }
  double v = 0.0;
  if (warp == 0 && ok) {
    v = a.f[f.col0 + k0 + lane];
    if (a.Dinv) v *= static_cast<double>(a.Dinv[f.col0 + k0 + lane]);
  }
  const T      *P    = a.panel + f.panel;
  const double *xr   = a.xr + (I.ticket % kFlowCopies) * a.n + f.col0;
  const int     cend = k0 + I.item.nr;
  float         lv[2][16], lvn[2][16];
  if (nsb - 1 > s) load_rows(lv, P, f.h, static_cast<int64_t>(nsb - 1) * kFlowSB,
                             w - (nsb - 1) * kFlowSB, k0, cend);
  flow_fetch(a, N);
  // Chunk partials: warp v takes chunks v, v + 16, .. of the slab's columns.
  double p2 = 0.0;
  if (ok)
    for (int c = warp; c < f.chunks; c += 16)
      p2 += wait_value(a.part + f.part + static_cast<int64_t>(c) * w + k0 + lane, a.err, polls);
  part[32 * warp + lane] = p2;
  double s0 = 0.0, s1 = 0.0;
  for (int R = nsb - 1; R > s; R--) {
    double   *xb = xs + (R & 1) * 512;
    const int g  = R * kFlowSB + tid;
    if (R - 1 > s) {
      load_rows(lvn, P, f.h, static_cast<int64_t>(R - 1) * kFlowSB, kFlowSB, k0, cend);
      xb[tid] = g < w ? wait_value(xr + g, a.err, polls) : 0.0;
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 16; i++) {
        const double xv = xb[lane + 32 * i];
        s0 += static_cast<double>(lv[0][i]) * xv;
        s1 += static_cast<double>(lv[1][i]) * xv;
      }
#pragma unroll
      for (int q = 0; q < 2; q++)
#pragma unroll
        for (int i = 0; i < 16; i++) lv[q][i] = lvn[q][i];
    } else {
      // the last tile, widened before its wait (see rows_apply)
      double ld[2][16];
#pragma unroll
      for (int q = 0; q < 2; q++)
#pragma unroll
        for (int i = 0; i < 16; i++) ld[q][i] = static_cast<double>(lv[q][i]);
      xb[tid] = g < w ? wait_value(xr + g, a.err, polls) : 0.0;
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 16; i++) {
        const double xv = xb[lane + 32 * i];
        s0 += ld[0][i] * xv;
        s1 += ld[1][i] * xv;
      }
    }
  }
  const double t2 = sum2(s0, s1);
  if ((lane & 15) == 0) ts2[2 * warp + (lane >> 4)] = t2;
  __syncthreads();
  double *xz = a.xz + f.col0 + s * kFlowSB;
  if (warp == 0) {
    double t[4] = {ts2[lane], 0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 16; q++) t[q % 4] += part[32 * q + lane];
    v = ok ? v - ((t[0] + t[1]) + (t[2] + t[3])) : 0.0;
    if (j > 0 && ok) st_relaxed_f64(xz + 32 * j + lane, v);
  }
  bulk_wait(bar, phase, a.err);
  phase ^= 1;
  if (j + warp < nsl) {
    const int     i   = j + warp;
    const double *blk = inv + warp * kFlowBlk + 33 * lane;
    double        iv[32];
#pragma unroll
    for (int r = 0; r < 32; r++) iv[r] = blk[r];
    if (warp > 0)
      v = s * kFlowSB + 32 * i + lane < w ? wait_value(xz + 32 * i + lane, a.err, polls) : 0.0;
    xs[32 * warp + lane] = v;
    __syncwarp();
    ts[32 * warp + lane] = dot32(iv, xs + 32 * warp);
  }
  __syncthreads();
  if (warp == 0 && ok) {
    double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 16; q++)
      if (j + q < nsl) t[q % 4] += ts[32 * q + lane];
    const double  xv = (t[0] + t[1]) + (t[2] + t[3]);
    const int64_t g  = f.col0 + k0 + lane;
#pragma unroll
    for (int c = 0; c < kFlowCopies; c++) st_relaxed_f64(a.xr + c * a.n + g, xv);
    a.x[g] = xv;
  }
}

// kFlowWarps, backward: t = the rows below, then x = Inv^T (z - t), lane =
// column (the panel's odd pitch keeps that free of bank conflicts; of fronts
// with at most 16 columns each half of the warp takes every other row).
template <class T>
__device__ __noinline__ void bwd_warp(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I, FlowSlot &N,
                                      double *sm, uint32_t &wphase) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  if (warp >= I.item.nr) {
    flow_fetch(a, N);
    return;
  }
  const long      polls = I.polls;
  const FlowFront f = a.warps[I.item.r0 + warp];
  const int       w = f.w, h = f.h, ld = h | 1, nr = h - w;
  const uint32_t  bar = smem_addr(&S.wbar[warp]);
  const double   *M   = warp_panel(a, f, sm, bar);
  constexpr int   RT = kWarpSolveH / 32;
  double         *vs = sm + kFlowInvSmem + 288 * warp, *xs = vs + 32;
  double          v  = 0.0;
  if (lane < w) {
    v = a.f[f.col0 + lane];
    if (a.Dinv) v *= static_cast<double>(a.Dinv[f.col0 + lane]);
  }
  {
    uint32_t gi[RT];
    double   xv[RT];
#pragma unroll
    for (int t = 0; t < RT; t++) {
      gi[t] = lane + 32 * t < nr ? static_cast<uint32_t>(a.srows[f.rows + w + lane + 32 * t]) : kFlowNone;
      xv[t] = 0.0;
    }
    flow_fetch(a, N);
    bulk_wait(bar, wphase, a.err);
    wphase ^= 1;
    wait_gate(a, f.gate, polls);
    add_values<RT>(a.xr, gi, xv, a.err, polls);
#pragma unroll
    for (int t = 0; t < RT; t++) xs[lane + 32 * t] = xv[t];
  }
  __syncwarp();
  const bool    half = w <= 16;
  const double *col  = M + min(half ? lane & 15 : lane, w - 1) * ld;
  const int     step = half ? 2 : 1;
  double        t0 = 0.0, t1 = 0.0, t2 = 0.0, t3 = 0.0;
  int           r  = half ? lane >> 4 : 0;
#pragma unroll 2
  for (; r + 3 * step < nr; r += 4 * step) {
    t0 += col[w + r] * xs[r];
    t1 += col[w + r + step] * xs[r + step];
    t2 += col[w + r + 2 * step] * xs[r + 2 * step];
    t3 += col[w + r + 3 * step] * xs[r + 3 * step];
  }
  for (; r < nr; r += step) t0 += col[w + r] * xs[r];
  double t = (t0 + t1) + (t2 + t3);
  if (half) t += __shfl_xor_sync(0xffffffffu, t, 16);
  vs[lane] = lane < w ? v - t : 0.0;
  __syncwarp();
  double x0 = 0.0, x1 = 0.0;
  int    i  = 0;
#pragma unroll 4
  for (; i + 1 < w; i += 2) {
    x0 += col[i] * vs[i];
    x1 += col[i + 1] * vs[i + 1];
  }
  if (i < w) x0 += col[i] * vs[i];
  if (lane < w) {
    st_relaxed_f64(a.xr + f.col0 + lane, x0 + x1);
    a.x[f.col0 + lane] = x0 + x1;
  }
}

template <class T>
__global__ void __launch_bounds__(kFlowThreads, 1) k_bwd_flow(const __grid_constant__ FlowArgs<T> a) {
  grid_wait();
  extern __shared__ __align__(128) double sm[];
  __shared__ __align__(16) FlowShared S;
  uint32_t phase = 0, wphase = 0;
  if (flow_idle(a)) return;
  flow_loop<false>(a, S, [&](const FlowSlot &I, FlowSlot &N) {
    switch (I.item.kind) {
      case kFlowWarps: bwd_warp(a, S, I, N, sm, wphase); break;
      case kBwdChunk: bwd_chunk(a, I, N, sm); break;
      case kBwdNarrow: bwd_narrow(a, S, I, N, sm, phase); break;
      default: bwd_slab(a, S, I, N, sm, phase);
    }
  });
  flow_mark(a.mark, a.nmark);
}

// ---------------------------------------------------------------------------
// Leaves of at most 64 rows (FlowFront, one warp each, lane = rows l and l + 32) by
// substitution with the float32 panel, for one vector, before the forward and after
// the backward data flow.  A front waits on nothing, so what bounds it is latency,
// and 64 warps an SM hide it where 16 with their fronts staged in shared memory do
// not.  One application by items, by levels before those, and so (ms): 10,000
// blocks of 40 x 40 0.40, 0.14, 0.08, 1,000 0.053, 0.043, 0.033; 100,000 of 4 x 4 0.22,
// 0.20, 0.11; 500,000 of one 0.99, 0.69, 0.33; 2-D grids of n = 640,000 0.52, 1.11, 0.44 and
// 250,000 0.25, 0.63, 0.24 (the line, kFlowLeafItems, where the items of a direction take
// about 15 us; below it two more launches weigh as much as they save).
constexpr int kLeafWarps = 8;
__global__ void __launch_bounds__(32 * kLeafWarps)
    k_fwd_leaf(const FlowFront *fronts, int count, const float *panel, const double *x, double *f,
               double *z, const int32_t *active) {
  grid_wait();
  if (active && *active == 0) return;
  const int lane = threadIdx.x % 32, q = blockIdx.x * kLeafWarps + threadIdx.x / 32;
  if (q >= count) return;
  const FlowFront fr = fronts[q];
  const int       w = fr.w, h = fr.h, i1 = lane + 32;
  const float    *P = panel + fr.panel;
  double          z0 = lane < w ? x[fr.col0 + lane] : 0.0, z1 = i1 < w ? x[fr.col0 + i1] : 0.0;
  float           c0[4], c1[4], n0[4], n1[4];
  auto            load = [&](float(&a)[4], float(&b)[4], int k0) {
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int k = k0 + u;
      a[u]        = k < w && lane > k && lane < h ? P[lane + k * h] : 0.0f;
      b[u]        = k < w && i1 > k && i1 < h ? P[i1 + k * h] : 0.0f;
    }
  };
  load(c0, c1, 0);
  for (int k0 = 0; k0 < w; k0 += 4) {
    load(n0, n1, k0 + 4);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int k = k0 + u;
      if (k >= w) break;
      const double y = __shfl_sync(0xffffffffu, k < 32 ? z0 : z1, k % 32);
      if (lane > k) z0 -= static_cast<double>(c0[u]) * y;
      if (i1 > k) z1 -= static_cast<double>(c1[u]) * y;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      c0[u] = n0[u];
      c1[u] = n1[u];
    }
  }
  if (lane < h) (lane < w ? f + fr.col0 : z + fr.zofs)[lane] = z0;
  if (i1 < h) (i1 < w ? f + fr.col0 : z + fr.zofs)[i1] = z1;
}

__global__ void __launch_bounds__(32 * kLeafWarps)
    k_bwd_leaf(const FlowFront *fronts, int count, const float *panel, const int32_t *srows,
               const float *Dinv, const double *f, double *x, const int32_t *active) {
  grid_wait();
  if (active && *active == 0) return;
  const int lane = threadIdx.x % 32, q = blockIdx.x * kLeafWarps + threadIdx.x / 32;
  if (q >= count) return;
  const FlowFront fr = fronts[q];
  const int       w = fr.w, h = fr.h, i1 = lane + 32;
  const float    *P  = panel + fr.panel;
  auto            at = [&](int i) {
    if (i >= h) return 0.0;
    if (i >= w) return x[srows[fr.rows + i]];
    return Dinv ? f[fr.col0 + i] * static_cast<double>(Dinv[fr.col0 + i]) : f[fr.col0 + i];
  };
  double x0 = at(lane), x1 = at(i1);
  float  c0[4], c1[4], n0[4], n1[4];
  auto   load = [&](float(&a)[4], float(&b)[4], int k0) {  // columns k0, k0 - 1, ..
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int k = k0 - u;
      a[u]        = k >= 0 && lane > k && lane < h ? P[lane + k * h] : 0.0f;
      b[u]        = k >= 0 && i1 > k && i1 < h ? P[i1 + k * h] : 0.0f;
    }
  };
  load(c0, c1, w - 1);
  for (int k0 = w - 1; k0 >= 0; k0 -= 4) {
    load(n0, n1, k0 - 4);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int k = k0 - u;
      if (k < 0) break;
      double s = lane > k ? static_cast<double>(c0[u]) * x0 : 0.0;
      if (i1 > k) s += static_cast<double>(c1[u]) * x1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == k) x0 -= s;
      if (i1 == k) x1 -= s;
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      c0[u] = n0[u];
      c1[u] = n1[u];
    }
  }
  if (lane < w) x[fr.col0 + lane] = x0;
  if (i1 < w) x[fr.col0 + i1] = x1;
}

__global__ void k_dscale(int64_t n, const float *Dinv, double *x) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) x[i] *= static_cast<double>(Dinv[i]);
}

// ---------------------------------------------------------------------------
// Inverses of the diagonal super-blocks in float64 from the float32 factor,
// once per factorization: a CTA of four warps solves L X = E for 16 columns, by
// blocks of 32 rows.  The block's triangle takes four columns a warp (lane =
// row, the pivots' values by shuffle); the block's columns then go into the
// sums of the rows below on the float64 matrix instructions, row block i on
// warp i mod 4.  What bounds it is the chain of up to 16 blocks and the
// float32 -> float64 conversions (24 cycles for a lone warp), which a fragment
// shares among 16 columns.  A warp with two columns of its own and a
// conversion for each use of L took 86 us for one block of 311 columns and 205
// us at n = 24,603; it is 38 and 114 us so (with eight warps 45 and 148).
constexpr int kInvCols  = 16;
constexpr int kInvPitch = 20;  // conflict-free fragments
__global__ void __launch_bounds__(128)
    k_flow_invert(const FlowInvDesc *descs, const float *panel, double *inv) {
  __shared__ __align__(16) double xs[32 * kInvPitch];  // X of the block: row, column
  __shared__ __align__(16) double as[32 * (kInvCols + 2)];  // its sum
  const FlowInvDesc d    = descs[blockIdx.x];
  const int         warp = threadIdx.x / 32, lane = threadIdx.x % 32, fr = lane / 4, fk = lane % 4;
  const int         n = d.n, nb = (n + 31) / 32, col = d.c0 + 4 * warp, j = d.c0 / 32;
  const int64_t     h = d.h;
  const float      *P = panel + d.panel;
  double            acc[4][4][2][2] = {};  // row block 4 slot + warp, octet, column octet
  for (int i = j; i < nb; i++) {
    const int row = 32 * i + lane;
    float     l[32];
    load_cols(l, P, h, row, row < n, 32 * i, min(n, 32 * i + lane));
#pragma unroll
    for (int s = 0; s < 4; s++)
      if (i == 4 * s + warp) {
#pragma unroll
        for (int m = 0; m < 4; m++)
#pragma unroll
          for (int q = 0; q < 2; q++)
            *reinterpret_cast<double2 *>(as + (8 * m + fr) * (kInvCols + 2) + 8 * q + 2 * fk) =
                make_double2(acc[s][m][q][0], acc[s][m][q][1]);
      }
    __syncthreads();
    double v[4];
#pragma unroll
    for (int u = 0; u < 4; u++)
      v[u] = (row == col + u && row < n ? 1.0 : 0.0) - as[lane * (kInvCols + 2) + 4 * warp + u];
#pragma unroll
    for (int k = 0; k < 32; k++) {
      const double lk = static_cast<double>(l[k]);
#pragma unroll
      for (int u = 0; u < 4; u++) v[u] -= lk * __shfl_sync(0xffffffffu, v[u], k);
    }
    double *o = inv + d.inv + (static_cast<int64_t>(i) * (i + 1) / 2 + j) * kFlowBlk + (col % 32) * 33 + lane;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      o[33 * u]                              = v[u];
      xs[lane * kInvPitch + 4 * warp + u] = v[u];
    }
    __syncthreads();
    if (i + 1 == nb) break;
    double b[8][2];
#pragma unroll
    for (int t = 0; t < 8; t++)
#pragma unroll
      for (int q = 0; q < 2; q++) b[t][q] = xs[(4 * t + fk) * kInvPitch + 8 * q + fr];
#pragma unroll
    for (int s = 0; s < 4; s++) {
      const int e = 4 * s + warp;
      if (e <= i || e >= nb) continue;
      const float *p = P + 32 * e + fr + (int64_t)(32 * i + fk) * h;
#pragma unroll
      for (int m = 0; m < 4; m++)
#pragma unroll
        for (int t = 0; t < 8; t++)
          l[8 * m + t] = 32 * e + 8 * m + fr < n ? __ldg(p + 8 * m + 4 * t * h) : 0.0f;
#pragma unroll
      for (int m = 0; m < 4; m++)
#pragma unroll
        for (int t = 0; t < 8; t++) {
          const double x = static_cast<double>(l[8 * m + t]);
#pragma unroll
          for (int q = 0; q < 2; q++)
            asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                : "+d"(acc[s][m][q][0]), "+d"(acc[s][m][q][1])
                : "d"(x), "d"(b[t][q]));
        }
    }
  }
}

// Panels of the warp-solved fronts in float64, the w x w triangle replaced by
// its inverse (zeros above the diagonal), columns h | 1 apart: one warp per
// front, lane = column of the inverse.  A conversion takes a lone warp 24
// cycles (measured, against 2 for an FMA): for a front of 256 x 32 that was
// 3 us of each solve; and with the inverse the block solve is a sum, not a
// chain of w steps.
__global__ void __launch_bounds__(128)
    k_flow_wpanel(const FlowFront *fronts, int count, const float *panel, double *wpanel) {
  __shared__ float ls[4][32][33];
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, q = 4 * blockIdx.x + warp;
  if (q >= count) return;
  const FlowFront f = fronts[q];
  const int       w = f.w, h = f.h, ld = h | 1;
  const float    *P = panel + f.panel;
  double         *M = wpanel + f.inv;
  for (int k = 0; k < w; k++) {
    for (int i = w + lane; i < h; i += 32) M[k * ld + i] = static_cast<double>(P[i + k * h]);
    ls[warp][lane][k] = lane > k && lane < w ? P[lane + k * h] : 0.0f;
  }
  __syncwarp();
  double x[32];
#pragma unroll
  for (int i = 0; i < 32; i++) {
    double s = i == lane ? 1.0 : 0.0;
    if (i < w) {
#pragma unroll
      for (int k = 0; k < i; k++) s -= static_cast<double>(ls[warp][i][k]) * x[k];
      if (lane < w) M[lane * ld + i] = s;
    }
    x[i] = s;
  }
}

void flow_invert(const Plan &P, Numeric &F, FlowPart part, cudaStream_t s) {
  // Warp-solved fronts: with the part that holds the last of them.
  const int32_t nw = static_cast<int32_t>(P.host_.flow_warp.size());
  if (nw > 0 && (part == kFlowAll || (part == kFlowTop) == P.flow_warp_top))
    launch(k_flow_wpanel, static_cast<unsigned>((nw + 3) / 4), 128, 0, s,
           static_cast<const FlowFront *>(P.flow_warp.as<FlowFront>()), nw,
           static_cast<const float *>(F.panel.as<float>()), F.wpanel.as<double>());
  const int32_t first = part == kFlowTop ? P.nflow_inv_low : 0;
  const int32_t count = (part == kFlowLow ? P.nflow_inv_low : P.nflow_inv) - first;
  if (count > 0)
    launch(k_flow_invert, static_cast<unsigned>(count), 128, 0, s,
           static_cast<const FlowInvDesc *>(P.flow_inv.as<FlowInvDesc>() + first),
           static_cast<const float *>(F.panel.as<float>()), F.inv64.as<double>());
  MPIR_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
namespace {
// The handed-over values in one buffer: the forward solve's, then the
// backward solve's (each side is marked pending as a whole).
struct FlowBuffers {
  int64_t fwd, bwd;
  explicit FlowBuffers(const Plan &P)
      : fwd(P.flow_z_elems + (kFlowCopies + 1) * P.S.n),
        bwd(P.flow_part_elems + (kFlowCopies + 1) * P.S.n) {}
};
}  // namespace

size_t SolveWorkspace::bytes_for(const Plan &P) {
  const FlowBuffers b(P);
  return (b.fwd + b.bwd + P.S.n) * sizeof(double) + 4 * sizeof(int32_t) + sizeof(SolveCtl);
}

void SolveWorkspace::allocate(const Plan &P) {
  const FlowBuffers b(P);
  vals.resize(std::max<int64_t>(b.fwd + b.bwd + P.S.n, 1) * sizeof(double));
  sync.resize(4 * sizeof(int32_t));
  device_zero(sync.as<void>(), sync.bytes());
  err.resize(sizeof(SolveCtl));
  device_zero(err.as<void>(), sizeof(SolveCtl));
  fwd_pending = bwd_pending = false;
  static OncePerDevice attr;
  allow_smem(attr, kFlowSmemBytes,
             {reinterpret_cast<const void *>(k_fwd_flow<float, false>),
              reinterpret_cast<const void *>(k_fwd_flow<float, true>),
              reinterpret_cast<const void *>(k_fwd_flow<__half, false>),
              reinterpret_cast<const void *>(k_fwd_flow<__half, true>),
              reinterpret_cast<const void *>(k_fwd_flow<__nv_bfloat16, false>),
              reinterpret_cast<const void *>(k_fwd_flow<__nv_bfloat16, true>),
              reinterpret_cast<const void *>(k_bwd_flow<float>),
              reinterpret_cast<const void *>(k_bwd_flow<__half>),
              reinterpret_cast<const void *>(k_bwd_flow<__nv_bfloat16>)});
}

template <class T>
static void ldlt_solve_t(const Plan &P, const Numeric &F, const T *pan, double *x,
                         SolveWorkspace &ws, cudaStream_t s, int phases, const ActiveFlags &act) {
  const int64_t n = P.S.n;
  if (n == 0) return;
  KernelTimer      &kt = kernel_timer();
  const FlowBuffers b(P);
  double           *fv = ws.vals.as<double>(), *bv = fv + b.fwd;
  FlowArgs<T> a{};
  a.warps = P.flow_warp.as<FlowFront>();
  a.panel = pan;
  a.inv   = F.inv64.as<double>();
  a.wpanel = F.wpanel.as<double>();
  a.gfirst = P.flow_gfirst.as<FlowGather>();
  a.gmore  = P.flow_gmore.as<uint32_t>();
  a.srows = P.srows.as<int32_t>();
  a.n     = n;
  a.x     = x;
  a.f     = (phases & kForward) ? bv + b.bwd : x;
  a.z     = fv;
  a.y     = a.z + P.flow_z_elems;
  a.yz    = a.y + kFlowCopies * n;
  a.part  = bv;
  a.xr    = a.part + P.flow_part_elems;
  a.xz    = a.xr + kFlowCopies * n;
  a.err   = ws.err.as<int32_t>();
  a.active        = act.p;
  a.nactive       = act.count;
  a.active_stride = act.stride;
  constexpr int smem = kFlowSmemBytes;
  // (The 16-bit panels are left to the items, which take these fronts' float32 values.
  // Beside the leaves' kernels there may be few items or none; the launch still marks
  // all the values pending.)
  const bool      leaf  = std::is_same<T, float>::value && P.nflow_leaf > 0;
  const FlowFront *lf   = P.flow_leaf.as<FlowFront>();
  const float     *lp   = F.panel.as<float>();
  const unsigned   lgrid = static_cast<unsigned>((P.nflow_leaf + kLeafWarps - 1) / kLeafWarps);
  kt.begin(kKcSolveFwd, s);
  if (phases & kForward) {
    if (!ws.fwd_pending) flow_pending(fv, b.fwd, s);
    if (leaf)
      launch_chained(n, k_fwd_leaf, 1, lgrid, 32 * kLeafWarps, 0, s, lf, P.nflow_leaf, lp, x, a.f, a.z, act.p);
    const int32_t skip = leaf ? P.nflow_leaf_fwd : 0;
    a.items  = P.flow_fwd.as<FlowItem>() + skip;
    a.nitems = P.nflow_fwd - skip;
    a.mark   = bv;
    a.nmark  = b.bwd;
    a.ticket = ws.sync.as<int32_t>();
    launch_chained(n, P.flow_z_elems > P.S.z_elems ? k_fwd_flow<T, true> : k_fwd_flow<T, false>, 1,
                   leaf ? kSMs : std::min(a.nitems, kSMs), kFlowThreads, smem, s, a);
    ws.fwd_pending = false;
    ws.bwd_pending = true;
  }
  if (!(phases & kBackward) && (phases & kForward))
    MPIR_CUDA(cudaMemcpyAsync(x, a.f, n * sizeof(double), cudaMemcpyDeviceToDevice, s));
  // The backward solve reads f .* Dinv as its right-hand side.
  if ((phases & kDiagonal) && !(phases & kBackward))
    launch(k_dscale, static_cast<unsigned>((n + 255) / 256), 256, 0, s, n, F.Dinv.as<float>(), x);
  kt.end(s);
  MPIR_CHECK_LAUNCH();
  if (!(phases & kBackward)) return;
  kt.begin(kKcSolveBwd, s);
  if (!ws.bwd_pending) flow_pending(bv, b.bwd, s);
  a.items  = P.flow_bwd.as<FlowItem>();
  a.nitems = P.nflow_bwd - (leaf ? P.nflow_leaf_bwd : 0);
  a.mark   = fv;
  a.nmark  = b.fwd;
  a.Dinv   = (phases & kDiagonal) ? F.Dinv.as<float>() : nullptr;
  a.ticket = ws.sync.as<int32_t>() + 1;
  launch_chained(n, k_bwd_flow<T>, 1, leaf ? kSMs : std::min(a.nitems, kSMs), kFlowThreads, smem, s, a);
  if (leaf)
    launch_chained(n, k_bwd_leaf, 1, lgrid, 32 * kLeafWarps, 0, s, lf, P.nflow_leaf, lp, a.srows, a.Dinv, a.f, x,
                   act.p);
  ws.bwd_pending = false;
  ws.fwd_pending = true;
  kt.end(s);
  MPIR_CHECK_LAUNCH();
}

void ldlt_solve(const Plan &P, const Numeric &F, double *x, SolveWorkspace &ws,
                cudaStream_t s, int phases, const ActiveFlags &act) {
  switch (F.solve_prec()) {
    case 2:
      ldlt_solve_t(P, F, F.panel16.as<__nv_bfloat16>(), x, ws, s, phases, act);
      break;
    case 3:
      ldlt_solve_t(P, F, F.panel16.as<__half>(), x, ws, s, phases, act);
      break;
    default:
      ldlt_solve_t(P, F, F.panel.as<float>(), x, ws, s, phases, act);
  }
}

// ---------------------------------------------------------------------------
// QDLDL_solve without device allocation.
//
// For callers that cannot call cudaMalloc: processes whose device memory is
// reserved up front and handed out entirely by their own pooling allocator,
// and loops that cannot take cudaMalloc's implicit device-wide
// synchronisation.  All
// device data of this entry point (the supernodal layout of L, the factor
// values, Dinv, the fronts' update vectors and x) is packed into the one
// file-scope array below, of fixed size, that every GPU holds once this
// library is loaded.  Only factors whose supernodal fronts have at most
// kSmallFront rows are taken (the warp-per-front kernels; no diagonal-block
// inverses), and the packed data must fit the array.
constexpr int kWarpsPerCta = 4;
constexpr int kSmallH      = kWarpSolveH;

// Forward
__global__ void __launch_bounds__(32 * kWarpsPerCta)
    k_fwd_small(const int32_t *list, int count, const int64_t *sfirst,
                const int64_t *srowptr, const int64_t *slofs,
                const int64_t *child_ptr, const int32_t *child_list,
                const int32_t *srel, const int64_t *zofs, const float *panel,
                double *x, double *zbuf) {
  __shared__ double zs[kWarpsPerCta][kSmallH];
  const int         warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int         idx  = blockIdx.x * kWarpsPerCta + warp;
  if (idx >= count) return;
  const int      J = list[idx];
  const int64_t  f = sfirst[J];
  const int      w = static_cast<int>(sfirst[J + 1] - f);
  const int      h = static_cast<int>(srowptr[J + 1] - srowptr[J]);
  double        *z = zs[warp];
  for (int i = lane; i < h; i += 32) z[i] = i < w ? x[f + i] : 0.0;
  __syncwarp();
  for (int64_t c = child_ptr[J]; c < child_ptr[J + 1]; c++) {
    const int      C  = child_list[c];
    const int      wc = static_cast<int>(sfirst[C + 1] - sfirst[C]);
    const int      rc = static_cast<int>(srowptr[C + 1] - srowptr[C]) - wc;
    const int32_t *rl = srel + srowptr[C] + wc;
    const double  *zc = zbuf + zofs[C] + wc;
    for (int a = lane; a < rc; a += 32) z[rl[a]] += zc[a];
    __syncwarp();
  }
  // Columns four at a time; the next four columns' entries of this lane's
  // rows (lane + 32 t) are loaded while the current four are applied.
  const float  *P  = panel + slofs[J];
  constexpr int RT = kSmallH / 32;
  float         cur[4][RT], nxt[4][RT];
  auto          load4 = [&](float (*buf)[RT], int k0) {
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int t = 0; t < RT; t++) {
        const int k = k0 + u, i = lane + 32 * t;
        buf[u][t]   = (k < w && i > k && i < h) ? P[i + (int64_t)k * h] : 0.0f;
      }
  };
  load4(cur, 0);
  for (int k0 = 0; k0 < w; k0 += 4) {
    if (k0 + 4 < w) load4(nxt, k0 + 4);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int k = k0 + u;
      if (k >= w) break;
      const double zk = z[k];
#pragma unroll
      for (int t = 0; t < RT; t++) {
        const int i = lane + 32 * t;
        if (i > k && i < h) z[i] -= static_cast<double>(cur[u][t]) * zk;
      }
      __syncwarp();
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int t = 0; t < RT; t++) cur[u][t] = nxt[u][t];
  }
  double *zo = zbuf + zofs[J];
  for (int i = lane; i < h; i += 32) {
    if (i < w) x[f + i] = z[i];
    zo[i] = z[i];
  }
}

// Backward
__global__ void __launch_bounds__(32 * kWarpsPerCta)
    k_bwd_small(const int32_t *list, int count, const int64_t *sfirst,
                const int64_t *srowptr, const int32_t *srows,
                const int64_t *slofs, const float *panel, double *x) {
  __shared__ double zs[kWarpsPerCta][kSmallH];
  const int         warp = threadIdx.x / 32, lane = threadIdx.x % 32;
  const int         idx  = blockIdx.x * kWarpsPerCta + warp;
  if (idx >= count) return;
  const int      J  = list[idx];
  const int64_t  f  = sfirst[J];
  const int      w  = static_cast<int>(sfirst[J + 1] - f);
  const int      h  = static_cast<int>(srowptr[J + 1] - srowptr[J]);
  const int32_t *rw = srows + srowptr[J];
  double        *z  = zs[warp];
  for (int i = lane; i < h; i += 32) z[i] = i < w ? x[f + i] : x[rw[i]];
  __syncwarp();
  // Columns four at a time from the last; the next four columns' entries of
  // this lane's rows (lane + 32 t) are loaded while the current four are used.
  const float  *P  = panel + slofs[J];
  constexpr int RT = kSmallH / 32;
  float         cur[4][RT], nxt[4][RT];
  auto          load4 = [&](float (*buf)[RT], int k0) {  // columns k0, k0-1, ..
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int t = 0; t < RT; t++) {
        const int k = k0 - u, i = lane + 32 * t;
        buf[u][t]   = (k >= 0 && i > k && i < h) ? P[i + (int64_t)k * h] : 0.0f;
      }
  };
  load4(cur, w - 1);
  for (int k0 = w - 1; k0 >= 0; k0 -= 4) {
    if (k0 - 4 >= 0) load4(nxt, k0 - 4);
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int k = k0 - u;
      if (k < 0) break;
      double s = 0.0;
#pragma unroll
      for (int t = 0; t < RT; t++) {
        const int i = lane + 32 * t;
        if (i > k && i < h) s += static_cast<double>(cur[u][t]) * z[i];
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == 0) z[k] -= s;
      __syncwarp();
    }
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int t = 0; t < RT; t++) cur[u][t] = nxt[u][t];
  }
  for (int i = lane; i < w; i += 32) x[f + i] = z[i];
}

namespace {
constexpr size_t kNoAllocScratchBytes = size_t{32} << 20;  // 32 MiB
constexpr int    kNoAllocMaxDevices   = 64;
}  // namespace

static __device__ __align__(256) unsigned char g_solve_scratch[kNoAllocScratchBytes];

namespace {
// Device address of g_solve_scratch on each device, looked up on the first
// call that uses that device (atomic: host threads may make their first
// calls at the same time; they store the same address).
std::atomic<void *> g_solve_scratch_addr[kNoAllocMaxDevices] = {};

// Restores the calling thread's current device on every return path.
struct DeviceRestore {
  int  saved = -1;
  DeviceRestore() {
    if (cudaGetDevice(&saved) != cudaSuccess) saved = -1;
  }
  ~DeviceRestore() {
    if (saved >= 0) cudaSetDevice(saved);
  }
};
}  // namespace

int qdldl_solve_noalloc(int64_t n, const int64_t *Lp, const int64_t *Li, const float *Lx,
                        const float *Dinv, double *x, int device, std::string &err) {
  if (n < 0 || device < 0 || device >= kNoAllocMaxDevices) {
    err = "invalid dimension or device";
    return kBadArgument;
  }
  if (n == 0) return kOk;
  Symbolic  S;
  const int rc = analyze_from_L(n, Lp, Li, S, err);
  if (rc != kOk) return rc;
  for (int64_t J = 0; J < S.ns; J++)
    if (S.h(J) > kSmallFront) {
      err = "a supernodal front has " + std::to_string(S.h(J)) + " rows; this entry point takes at most " +
            std::to_string(kSmallFront);
      return -7;
    }
  // Factor values in the panel layout (explicit zeros for padding).
  std::vector<float> pan(S.panel_elems, 0.0f);
  for (int64_t J = 0; J < S.ns; J++) {
    const int64_t f = S.sfirst[J], l = S.sfirst[J + 1], w = l - f, h = S.h(J);
    for (int64_t j = f; j < l; j++) {
      int64_t q = S.srowptr[J] + w;  // rows below the supernode's own columns
      for (int64_t p = Lp[j]; p < Lp[j + 1]; p++) {
        const int64_t r = Li[p];
        int64_t       lr;
        if (r < l) {
          lr = r - f;
        } else {
          while (S.srows[q] < r) q++;
          lr = w + (q - S.srowptr[J] - w);
        }
        pan[S.slofs[J] + (j - f) * h + lr] = Lx[p];
      }
    }
  }
  // Pack every region into the scratch array, 256-byte aligned.
  struct Region {
    const void *src;
    size_t      bytes;
    size_t      ofs;
  };
  std::vector<Region> reg;
  size_t              top = 0;
  auto add = [&](const void *src, size_t bytes) {
    top = (top + 255) / 256 * 256;
    reg.push_back({src, bytes, top});
    top += bytes;
    return reg.size() - 1;
  };
  const size_t r_sfirst = add(S.sfirst.data(), S.sfirst.size() * sizeof(int64_t));
  const size_t r_srowptr = add(S.srowptr.data(), S.srowptr.size() * sizeof(int64_t));
  const size_t r_srows = add(S.srows.data(), S.srows.size() * sizeof(int32_t));
  const size_t r_srel = add(S.srel.data(), S.srel.size() * sizeof(int32_t));
  const size_t r_slofs = add(S.slofs.data(), S.slofs.size() * sizeof(int64_t));
  const size_t r_cptr = add(S.child_ptr.data(), S.child_ptr.size() * sizeof(int64_t));
  const size_t r_clist = add(S.child_list.data(), S.child_list.size() * sizeof(int32_t));
  const size_t r_zofs = add(S.zofs.data(), S.zofs.size() * sizeof(int64_t));
  const size_t r_level = add(S.level_sup.data(), S.level_sup.size() * sizeof(int32_t));
  const size_t r_panel = add(pan.data(), pan.size() * sizeof(float));
  const size_t r_dinv = add(Dinv, n * sizeof(float));
  const size_t r_x = add(x, n * sizeof(double));
  const size_t r_zbuf = add(nullptr, S.z_elems * sizeof(double));  // written on the device
  if (top > kNoAllocScratchBytes) {
    err = "needs " + std::to_string(top) + " bytes of device scratch; this entry point has " +
          std::to_string(kNoAllocScratchBytes);
    return kBadArgument;
  }
  DeviceRestore restore;  // the caller's current device is left as it was
  MPIR_CUDA(cudaSetDevice(device));
  void *addr = g_solve_scratch_addr[device].load(std::memory_order_acquire);
  if (!addr) {
    const cudaError_t e = cudaGetSymbolAddress(&addr, g_solve_scratch);
    if (e != cudaSuccess) throw CudaError(e, "cudaGetSymbolAddress(g_solve_scratch)");
    g_solve_scratch_addr[device].store(addr, std::memory_order_release);
  }
  unsigned char     *base = static_cast<unsigned char *>(addr);
  const cudaStream_t s    = cudaStreamPerThread;
  for (const Region &r : reg)
    if (r.src && r.bytes)
      MPIR_CUDA(cudaMemcpyAsync(base + r.ofs, r.src, r.bytes, cudaMemcpyHostToDevice, s));
  auto at = [&](size_t i) { return static_cast<void *>(base + reg[i].ofs); };
  const int64_t *sfirst  = static_cast<const int64_t *>(at(r_sfirst));
  const int64_t *srowptr = static_cast<const int64_t *>(at(r_srowptr));
  const int32_t *srows   = static_cast<const int32_t *>(at(r_srows));
  const int32_t *srel    = static_cast<const int32_t *>(at(r_srel));
  const int64_t *slofs   = static_cast<const int64_t *>(at(r_slofs));
  const int64_t *cptr    = static_cast<const int64_t *>(at(r_cptr));
  const int32_t *clist   = static_cast<const int32_t *>(at(r_clist));
  const int64_t *zofs    = static_cast<const int64_t *>(at(r_zofs));
  const int32_t *level   = static_cast<const int32_t *>(at(r_level));
  const float   *panel   = static_cast<const float *>(at(r_panel));
  const float   *dinv    = static_cast<const float *>(at(r_dinv));
  double        *xd      = static_cast<double *>(at(r_x));
  double        *zbuf    = static_cast<double *>(at(r_zbuf));
  const int      nl      = S.nlevels;
  for (int t = 0; t < nl; t++) {
    const int32_t cnt = static_cast<int32_t>(S.level_ptr[t + 1] - S.level_ptr[t]);
    launch(k_fwd_small, (cnt + kWarpsPerCta - 1) / kWarpsPerCta, 32 * kWarpsPerCta, 0, s,
           level + S.level_ptr[t], cnt, sfirst, srowptr, slofs, cptr, clist, srel, zofs, panel,
           xd, zbuf);
  }
  launch(k_dscale, static_cast<unsigned>((n + 255) / 256), 256, 0, s, n, dinv, xd);
  for (int t = nl - 1; t >= 0; t--) {
    const int32_t cnt = static_cast<int32_t>(S.level_ptr[t + 1] - S.level_ptr[t]);
    launch(k_bwd_small, (cnt + kWarpsPerCta - 1) / kWarpsPerCta, 32 * kWarpsPerCta, 0, s,
           level + S.level_ptr[t], cnt, sfirst, srowptr, srows, slofs, panel, xd);
  }
  MPIR_CHECK_LAUNCH();
  MPIR_CUDA(cudaMemcpyAsync(x, xd, n * sizeof(double), cudaMemcpyDeviceToHost, s));
  MPIR_CUDA(cudaStreamSynchronize(s));
  return kOk;
}

}  // namespace mpir
