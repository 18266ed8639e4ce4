// Triangular solves with several right-hand sides at once:
// X <- L^{-T} D^{-1} L^{-1} X for an n x NR block X (column-major, leading
// dimension n), the operation QDLDL_solve applies to one vector
// (qdldl.hpp:417-432) and LUIR_QDLDL / PrecondGmres apply once per vector.
//
// The work items, their order and the hand-over of values are those of the
// single-vector solves (solve.cu, flow.cuh): one launch a direction for the
// whole tree.  Each item takes all NR vectors: L moves once per application
// instead of NR times, and the hand-overs on the chain from the leaves to the
// root are shared by the NR vectors.  Between items the NR values of an entry
// lie side by side (entry i at NR i), so that a hand-over is NR / 2 loads of 16
// bytes; in shared memory too, where a warp reads the same entry's values for
// NR fused multiply-adds a value of L.
//
// Products with L and with the inverses run on the float64 matrix
// instructions (m8n8k4): a warp takes 32 x 32 entries of L, each lane those of
// its fragments, and a value of y from shared memory serves 8 multiply-adds a
// lane.  With plain FMAs, a read of 16 bytes for every 2, the reads took most
// of a wide front's time (16 vectors: 17 us per 512 columns of the root).
//
// What bounds it: below the root the chain of hand-overs, as for one vector;
// in the wide fronts the float64 multiply-adds (512 x 32 x 16 take 2.2 us of an
// SM, twice per 512 columns of the chain).
// Measured, one application, against the solves by levels that these replaced
// and, in between, the same items with plain FMAs: 16 vectors at n = 20,480:
// 0.48 ms (2.73; 0.64 to 0.78), 8 at n = 40,960: 0.80 ms (2.99; 0.95), 4 at
// n = 40,951: 0.46 ms (1.51; 0.44), for which half of each product is unused.
// Per vector the sums inside an item run in another order than in the
// single-vector kernels, so results agree with NR single solves to rounding.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "engine.hpp"
#include "solve.hpp"
#include "solve_dev.cuh"
#include "flow_dev.cuh"

namespace mpir {

void flow_pending(double *p, int64_t n, cudaStream_t s);

namespace {

constexpr int kMultiCopies = 2;  // copies of a wide front's block results

// Shared memory (doubles): kFlowInvSmem, then vectors and partial sums.  The
// most is taken by the backward solve of a narrow front with its rows below: 10
// blocks of the inverse, 512 + 128 + 256 entries of 16 values at a pitch of 18
// (of 8 values at a pitch of 10: 512 + 128 + 512).
constexpr int kMultiSmem = 10 * kFlowBlk + 896 * 18;
static_assert(kMultiSmem >= kFlowInvSmem + 512 * 18, "16 warps' 32 entries behind the inverse blocks");

// Narrow fronts stage at most 10 blocks of the inverse; their vectors start
// behind those.
constexpr int kNarrowInv = 10 * kFlowBlk;

// In shared memory an entry's NR values lie every NR + 2 doubles where the lanes
// of a warp read or write an entry each (16-byte accesses then go without bank
// conflicts; at a pitch of NR = 16 each took 8 times as long).
template <int NR>
constexpr int kPitch = NR + 2;

struct alignas(16) V2 {
  unsigned long long a, b;
};
__device__ __forceinline__ V2 ld_relaxed_2(const double *p) {
  V2 v;
  asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_2(double *p, double a, double b) {
  asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(__double_as_longlong(a)),
               "l"(__double_as_longlong(b))
               : "memory");
}

// Waits for K values side by side (16-byte aligned; none when !on) and adds
// them to v.  All are asked for at once; while they are pending, the last pair
// alone is polled (an entry's values are stored together): with 16 vectors the
// CTAs that wait on a wide front's newest results would otherwise poll 64 KB
// each.
template <int K>
__device__ __forceinline__ void add_entry(const double *p, bool on, double (&v)[K], int32_t *err,
                                          long polls) {
  unsigned need = on ? (1u << (K / 2)) - 1 : 0u;
  for (long it = 0; need != 0; it++) {
    V2 raw[K / 2];
    if (K > 2 && it > 0 && need >> (K / 2 - 1) != 0) {
      const V2 g = ld_relaxed_2(p + K - 2);
      if (g.a == kPending || g.b == kPending) {
        if (it >= polls) {
          atomicExch(err, 1);
          return;
        }
        if ((it & 63) == 63) {
          if (*reinterpret_cast<volatile int32_t *>(err) != 0) return;
          __nanosleep(32);
        }
        continue;
      }
    }
#pragma unroll
    for (int q = 0; q < K / 2; q++) {
      raw[q] = V2{kPending, kPending};
      if (need >> q & 1u) raw[q] = ld_relaxed_2(p + 2 * q);
    }
#pragma unroll
    for (int q = 0; q < K / 2; q++)
      if (raw[q].a != kPending && raw[q].b != kPending) {
        v[2 * q] += __longlong_as_double(static_cast<long long>(raw[q].a));
        v[2 * q + 1] += __longlong_as_double(static_cast<long long>(raw[q].b));
        need &= ~(1u << q);
      }
    if (need != 0 && it >= polls) {
      atomicExch(err, 1);
      return;
    }
    if ((it & 63) == 63) {
      if (*reinterpret_cast<volatile int32_t *>(err) != 0) return;
      __nanosleep(32);
    }
  }
}

// An entry's K values (zeros when !on) into shared memory.
template <int K>
__device__ __forceinline__ void get_entry(const double *p, bool on, double *dst, int32_t *err,
                                          long polls) {
  double v[K];
#pragma unroll
  for (int k = 0; k < K; k++) v[k] = 0.0;
  add_entry<K>(p, on, v, err, polls);
#pragma unroll
  for (int k = 0; k < K; k += 2) *reinterpret_cast<double2 *>(dst + k) = make_double2(v[k], v[k + 1]);
}

// acc[k] += l y[k] for the NR values at y (shared memory, 16-byte aligned).
template <int NR>
__device__ __forceinline__ void fma_entry(double l, const double *y, double (&acc)[NR]) {
#pragma unroll
  for (int q = 0; q < NR; q += 2) {
    const double2 v = *reinterpret_cast<const double2 *>(y + q);
    acc[q] += l * v.x;
    acc[q + 1] += l * v.y;
  }
}

template <int NR>
__device__ __forceinline__ void put_entry(double *dst, const double (&v)[NR]) {
#pragma unroll
  for (int k = 0; k < NR; k += 2) *reinterpret_cast<double2 *>(dst + k) = make_double2(v[k], v[k + 1]);
}

// A warp's 32 x NR result in fragments of the m8n8k4 product: c[o][n] holds, of
// row (lane / 4) of octet o, the vectors 8 n + 2 (lane % 4) and the next (of 4
// vectors half of the fragment is not used).
template <int NR>
struct Frag {
  static constexpr int kN = NR < 8 ? 1 : NR / 8;
  double               c[4][kN][2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int o = 0; o < 4; o++)
#pragma unroll
      for (int n = 0; n < kN; n++) c[o][n][0] = c[o][n][1] = 0.0;
  }
  // The lane's values of the entry at p (8 vectors a fragment).
  static __device__ __forceinline__ void get_b(double (&b)[kN], const double *p) {
    const int v = threadIdx.x % 32 / 4;
#pragma unroll
    for (int n = 0; n < kN; n++) b[n] = p[8 * n + (NR < 8 ? v % 4 : v)];
  }
  __device__ __forceinline__ void mma(int o, double a, const double (&b)[kN]) {
#pragma unroll
    for (int n = 0; n < kN; n++)
      asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
          : "+d"(c[o][n][0]), "+d"(c[o][n][1])
          : "d"(a), "d"(b[n]));
  }
  // Row of octet o held by the lane: 8 o + lane / 4, or (kPerm) 4 (lane / 4) + o.
  template <bool kPerm>
  static __device__ __forceinline__ int row(int o) {
    const int g = threadIdx.x % 32 / 4;
    return kPerm ? 4 * g + o : 8 * o + g;
  }
  template <bool kPerm>
  __device__ __forceinline__ void put(double *dst) const {
    const int v = 2 * (threadIdx.x % 4);
    if (NR < 8 && v >= 4) return;
#pragma unroll
    for (int o = 0; o < 4; o++)
#pragma unroll
      for (int n = 0; n < kN; n++)
        *reinterpret_cast<double2 *>(dst + kPitch<NR> * row<kPerm>(o) + 8 * n + v) =
            make_double2(c[o][n][0], c[o][n][1]);
  }
  __device__ __forceinline__ void add(const double *src) {
    const int v = 2 * (threadIdx.x % 4);
    if (NR < 8 && v >= 4) return;
#pragma unroll
    for (int o = 0; o < 4; o++)
#pragma unroll
      for (int n = 0; n < kN; n++) {
        const double2 s =
            *reinterpret_cast<const double2 *>(src + kPitch<NR> * row<false>(o) + 8 * n + v);
        c[o][n][0] += s.x;
        c[o][n][1] += s.y;
      }
  }
};

// Fragments of 32 x 32 entries of L: of L itself (rows rb .., columns c ..; row
// 8 o + lane / 4, column 4 q + lane % 4 in d[8 o + q]), or of its transpose
// (column 8 o + lane / 4, row 4 q + lane % 4).
template <class T>
__device__ __forceinline__ void load_frag(float (&d)[32], const T *P, int64_t h, int64_t rb, int64_t rend,
                                          int c, int cend) {
  const int     lane = threadIdx.x % 32;
  const int64_t r    = rb + lane / 4;
  const int     c0   = c + lane % 4;
  const T      *p    = P + r + c0 * h;
#pragma unroll
  for (int q = 0; q < 8; q++)
#pragma unroll
    for (int o = 0; o < 4; o++)
      d[8 * o + q] = (r + 8 * o < rend && c0 + 4 * q < cend) ? to_f(__ldg(p + 8 * o + 4 * q * h)) : 0.0f;
}
template <class T>
__device__ __forceinline__ void load_frag_t(float (&d)[32], const T *P, int64_t h, int64_t rb, int64_t rend,
                                            int c, int cend) {
  const int     lane = threadIdx.x % 32;
  const int64_t r    = rb + lane % 4;
  const int     c0   = c + lane / 4;
  const T      *p    = P + r + c0 * h;
#pragma unroll
  for (int o = 0; o < 4; o++)
#pragma unroll
    for (int q = 0; q < 8; q++)
      d[8 * o + q] = (r + 4 * q < rend && c0 + 8 * o < cend) ? to_f(__ldg(p + 4 * q + 8 * o * h)) : 0.0f;
}

// f += (32 x 32 entries of L) times the 32 entries at y.
template <int NR>
__device__ __forceinline__ void mma_tile(Frag<NR> &f, const float (&d)[32], const double *y) {
#pragma unroll
  for (int q = 0; q < 8; q++) {
    double b[Frag<NR>::kN];
    Frag<NR>::get_b(b, y + kPitch<NR> * (4 * q + threadIdx.x % 4));
#pragma unroll
    for (int o = 0; o < 4; o++) f.mma(o, static_cast<double>(d[8 * o + q]), b);
  }
}

// f = a 32 x 32 block of the inverse (entry (r, c) at 33 c + r) times the 32
// entries at y; rows as Frag::row<true>, which keeps the lanes' reads of the
// block free of bank conflicts.
template <int NR>
__device__ __forceinline__ void mma_inverse(Frag<NR> &f, const double *blk, const double *y) {
  const int g = threadIdx.x % 32 / 4, k = threadIdx.x % 4;
  f.zero();
#pragma unroll
  for (int q = 0; q < 8; q++) {
    double b[Frag<NR>::kN];
    Frag<NR>::get_b(b, y + kPitch<NR> * (4 * q + k));
#pragma unroll
    for (int o = 0; o < 4; o++) f.mma(o, blk[33 * (4 * q + k) + 4 * g + o], b);
  }
}
// f += its transpose times the 32 entries at y (the block's rows are taken in
// the order 16 (q / 4) + 4 k + q % 4, for the same reason).
template <int NR>
__device__ __forceinline__ void mma_inverse_t(Frag<NR> &f, const double *blk, const double *y) {
  const int g = threadIdx.x % 32 / 4, k = threadIdx.x % 4;
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const int r = 16 * (q / 4) + 4 * k + q % 4;
    double    b[Frag<NR>::kN];
    Frag<NR>::get_b(b, y + kPitch<NR> * r);
#pragma unroll
    for (int o = 0; o < 4; o++) f.mma(o, blk[33 * (8 * o + g) + r], b);
  }
}

// ---------------------------------------------------------------------------
// Forward.

// f += L(rb .., c) y_c over the columns c < cend of a wide front, tile by tile
// as the block results become ready (rows_apply of solve.cu); own: the warp's
// 32 entries of shared memory.
template <int RG, int NR, class T>
__device__ __forceinline__ void rows_apply_m(const FlowArgs<T> &a, const T *P, int64_t h, int64_t rb,
                                             int64_t rend, int cend, const double *y, double *own,
                                             Frag<NR> &f, long polls) {
  constexpr int TW = 512 / RG;
  const int     warp = threadIdx.x / 32, lane = threadIdx.x % 32, cq = 32 * (warp / RG);
  float         lv[32], lvn[32];
  load_frag(lv, P, h, rb, rend, cq, cend);
  for (int c = cq; c - cq < cend; c += TW) {
    if (c - cq + TW < cend) load_frag(lvn, P, h, rb, rend, c + TW, cend);
    get_entry<NR>(y + static_cast<int64_t>(NR) * (c + lane), c + lane < cend, own + kPitch<NR> * lane, a.err,
                  polls);
    __syncwarp();
    mma_tile(f, lv, own);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 32; k++) lv[k] = lvn[k];
  }
}

template <int NR, class T>
__device__ __noinline__ void fwd_slab_m(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I, FlowSlot &N,
                                        double *sm, uint32_t &phase) {
  const FlowFront &f   = I.item.f;
  const int        tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  constexpr int    NP  = kPitch<NR>;
  const int        row = tid / NR, v = tid % NR, at = NP * row + v;  // the thread's output, tid < 32 NR
  const long       polls = I.polls;
  const int        r0 = I.item.r0, s = r0 / kFlowSB, i = (r0 % kFlowSB) / 32;
  const bool       mine = row < I.item.nr, last = r0 + 32 >= f.w || i == 15;
  double          *inv = sm, *yw = sm + kFlowInvSmem, *own = yw + 32 * NP * warp;
  const uint32_t   bar = smem_addr(&S.bar);
  if (tid == 0) {
    const uint32_t bytes = (i + 1) * kFlowBlk * sizeof(double);
    bulk_expect(bar, bytes);
    bulk_get(inv, a.inv + f.inv + (static_cast<int64_t>(s) * kFlowTriSB + i * (i + 1) / 2) * kFlowBlk,
             bytes, bar);
  }
  flow_fetch(a, N);
  double zr = 0.0;
  if (mine) {
    Gather<NR> g;
    g.begin(a, f.zofs + r0 + row, a.z + v);
    zr = g.finish(a, a.z + v, a.x[v * a.n + f.col0 + r0 + row], polls);
  }
  Frag<NR> fr;
  if (s > 0) {
    fr.zero();
    rows_apply_m<1, NR>(a, a.panel + f.panel, f.h, r0, r0 + I.item.nr, s * kFlowSB,
                        a.y + ((I.ticket % kMultiCopies) * a.n + f.col0) * NR, own, fr, polls);
    fr.template put<false>(own);
    __syncthreads();
    if (row < 32) {
      double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int q = 0; q < 16; q++) t[q % 4] += yw[32 * NP * q + at];
      zr -= (t[0] + t[1]) + (t[2] + t[3]);
    }
    __syncthreads();
  }
  double *yz = a.yz + static_cast<int64_t>(NR) * (f.col0 + s * kFlowSB);
  if (row < 32) {
    if (!last && I.publish) st_relaxed_f64(yz + 32 * NR * i + tid, zr);
    yw[at] = zr;  // the diagonal block's, for warp 0
  }
  __syncthreads();
  bulk_wait(bar, phase, a.err);
  phase ^= 1;
  if (warp <= i) {
    const int j = warp == 0 ? i : warp - 1;
    if (warp > 0) get_entry<NR>(yz + NR * (32 * j + lane), true, own + NP * lane, a.err, polls);
    __syncwarp();
    mma_inverse(fr, inv + j * kFlowBlk, own);
    __syncwarp();
    fr.template put<true>(own);
  }
  __syncthreads();
  if (mine) {
    double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 16; q++)
      if (q <= i) t[q % 4] += yw[32 * NP * q + at];
    const double  y = (t[0] + t[1]) + (t[2] + t[3]);
    const int64_t g = static_cast<int64_t>(NR) * (f.col0 + r0) + tid;
    if (I.publish) {
#pragma unroll
      for (int c = 0; c < kMultiCopies; c++) st_relaxed_f64(a.y + c * a.n * NR + g, y);
    }
    a.f[g] = y;
  }
}

template <int NR, class T>
__device__ __noinline__ void fwd_rows_m(const FlowArgs<T> &a, const FlowSlot &I, FlowSlot &N, double *sm) {
  const FlowFront &f   = I.item.f;
  const int        tid = threadIdx.x, warp = tid / 32;
  const long       polls = I.polls;
  const int        r0 = I.item.r0, nr = I.item.nr;
  double          *yw = sm + kFlowInvSmem, *own = yw + 32 * kPitch<NR> * warp;
  flow_fetch(a, N);
  Frag<NR> fr;
  fr.zero();
  rows_apply_m<4, NR>(a, a.panel + f.panel, f.h, r0 + 32 * (warp % 4), r0 + nr, f.w,
                      a.y + ((I.ticket % kMultiCopies) * a.n + f.col0) * NR, own, fr, polls);
  fr.template put<false>(own);
  // Output e: row e / NR, vector e % NR; its column quarters are 4 warps apart.
  constexpr int KO = NR / 4;
  Gather<NR>    g[KO];
#pragma unroll
  for (int m = 0; m < KO; m++) {
    const int e = tid + 512 * m;
    if (e / NR < nr) g[m].begin(a, f.zofs + r0 + e / NR, a.z + e % NR);
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < KO; m++) {
    const int e = tid + 512 * m;
    if (e / NR < nr) {
      constexpr int NP = kPitch<NR>;
      const double *p = yw + NP * (e / NR) + e % NR;
      const double  t = (p[0] + p[128 * NP]) + (p[256 * NP] + p[384 * NP]);
      const double  u = g[m].finish(a, a.z + e % NR, 0.0, polls) - t;
      if (I.publish) st_relaxed_f64(a.z + NR * (f.zofs + r0) + e, u);
    }
  }
}

template <int RG, int NR, class T>
__device__ __noinline__ void fwd_narrow_m(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I,
                                          FlowSlot &N, double *sm, uint32_t &phase) {
  const FlowFront &f   = I.item.f;
  const int        tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int        w = f.w, nbw = (w + 31) / 32, nr = I.item.nr;
  const long       polls = I.polls;
  constexpr int    KO = NR / 4, NP = kPitch<NR>;
  double          *inv = sm, *zs = sm + kNarrowInv, *ys = zs + 128 * NP, *part = ys + 128 * NP;
  const uint32_t   bar = smem_addr(&S.bar);
  if (tid == 0) {
    const uint32_t bytes = nbw * (nbw + 1) / 2 * kFlowBlk * sizeof(double);
    bulk_expect(bar, bytes);
    bulk_get(inv, a.inv + f.inv, bytes, bar);
  }
  constexpr int kTile = 32 * RG;
  const int     cq = warp / RG, rw = 32 * (warp % RG);  // the warp's columns, rows of a tile
  const int64_t r0 = I.item.r0;
  const T      *P  = a.panel + f.panel;
  float         lv[32], lvn[32];
  load_frag(lv, P, f.h, r0 + rw, r0 + nr, 32 * cq, w);
  flow_fetch(a, N);
  {
    Gather<NR> g[KO];
#pragma unroll
    for (int m = 0; m < KO; m++) {
      const int e = tid + 512 * m;
      if (e < w * NR) g[m].begin(a, f.zofs + e / NR, a.z + e % NR);
    }
#pragma unroll
    for (int m = 0; m < KO; m++) {
      const int e = tid + 512 * m;
      if (e < 128 * NR)
        zs[NP * (e / NR) + e % NR] =
            e < w * NR ? g[m].finish(a, a.z + e % NR, a.x[(e % NR) * a.n + f.col0 + e / NR], polls)
                           : 0.0;
    }
  }
  __syncthreads();
  bulk_wait(bar, phase, a.err);
  phase ^= 1;
  // y = Inv z: warp 4 i + j takes block (i, j)
  const int bi = warp / 4, bj = warp % 4;
  Frag<NR>  fr;
  if (bi < nbw && bj <= bi) {
    mma_inverse(fr, inv + (bi * (bi + 1) / 2 + bj) * kFlowBlk, zs + 32 * NP * bj);
    fr.template put<true>(part + NP * (128 * bj + 32 * bi));
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < KO; m++) {
    const int e = tid + 512 * m, row = e / NR;
    if (e >= 128 * NR) break;
    double y = 0.0;
    if (row < w)
      for (int j = 0; j <= row / 32; j++) y += part[NP * (128 * j + row) + e % NR];
    ys[NP * row + e % NR] = y;
    if (row < w && r0 == w) a.f[static_cast<int64_t>(NR) * f.col0 + e] = y;
  }
  __syncthreads();
  for (int q = 0; q * kTile < nr; q++) {
    if ((q + 1) * kTile < nr) load_frag(lvn, P, f.h, r0 + (q + 1) * kTile + rw, r0 + nr, 32 * cq, w);
    fr.zero();
    mma_tile(fr, lv, ys + NP * 32 * cq);
    double *out = part + NP * (kTile * cq + rw);
    fr.template put<false>(out);
    if (RG == 16) {
      // one tile; the lane's row: its children's values, then the result
      __syncwarp();
      const int rt = rw + lane;
      if (rt < nr) {
        double u[NR];
#pragma unroll
        for (int k = 0; k < NR; k++) u[k] = -out[NP * lane + k];
        const FlowGather g = a.gfirst[f.zofs + r0 + rt];
        add_entry<NR>(a.z + static_cast<int64_t>(NR) * g.first, g.first != kFlowNone, u, a.err, polls);
        if (g.more != kFlowNone) {
          const uint32_t *m = a.gmore + g.more;
          for (uint32_t e = 1, n = m[0]; e <= n; e++)
            add_entry<NR>(a.z + static_cast<int64_t>(NR) * m[e], true, u, a.err, polls);
        }
        if (I.publish) {
          double *z = a.z + NR * (f.zofs + r0 + rt);
#pragma unroll
          for (int k = 0; k < NR; k += 2) st_relaxed_2(z + k, u[k], u[k + 1]);
        }
      }
    } else {
      Gather<NR> g[KO];
      const int  base = q * kTile * NR;  // output e of the item: row e / NR
#pragma unroll
      for (int m = 0; m < KO; m++) {
        const int e = base + tid + 512 * m;
        if (e / NR < nr) g[m].begin(a, f.zofs + r0 + e / NR, a.z + e % NR);
      }
      __syncthreads();
#pragma unroll
      for (int m = 0; m < KO; m++) {
        const int e = base + tid + 512 * m;
        if (e / NR < nr) {
          const double *p = part + NP * (e / NR - q * kTile) + e % NR;
          const double  t = (p[0] + p[128 * NP]) + (p[256 * NP] + p[384 * NP]);
          const double  u = g[m].finish(a, a.z + e % NR, 0.0, polls) - t;
          if (I.publish) st_relaxed_f64(a.z + NR * (f.zofs + r0) + e, u);
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < 32; k++) lv[k] = lvn[k];
  }
}

// kFwdSum: a thread a sum and vector, eight contributions at a time.
template <int NR, class T>
__device__ __noinline__ void fwd_sum_m(const FlowArgs<T> &a, const FlowSlot &I, FlowSlot &N) {
  flow_fetch(a, N);
  const int e = threadIdx.x / NR, v = threadIdx.x % NR;
  if (e >= I.item.nr) return;
  const uint32_t *m = a.gmore + I.item.f.rows + kFlowFan * e;
  const double   *z = a.z + v;
  double          s = 0.0;
  for (int q = 0; q < kFlowFan; q += 8) {
    uint32_t           idx[8];
    unsigned long long raw[8];
#pragma unroll
    for (int u = 0; u < 8; u++) idx[u] = m[q + u];
#pragma unroll
    for (int u = 0; u < 8; u++)
      raw[u] = idx[u] != kFlowNone ? ld_relaxed_u64(z + static_cast<int64_t>(NR) * idx[u]) : 0ull;
#pragma unroll
    for (int u = 0; u < 8; u++)
      if (idx[u] != kFlowNone)
        s += take_value(raw[u], z + static_cast<int64_t>(NR) * idx[u], a.err, I.polls);
  }
  if (I.publish) st_relaxed_f64(a.z + NR * (I.item.f.zofs + e) + v, s);
}

// The panels of an item's warp-solved fronts into shared memory: warp q starts
// the copy of front q.
template <class T>
__device__ __forceinline__ void panels_get(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I,
                                           double *sm) {
  const int warp = threadIdx.x / 32;
  if (warp < I.item.nr) warp_panel(a, a.warps[I.item.r0 + warp], sm, smem_addr(&S.wbar[warp]));
}

// kFlowWarps: two vectors of a front per warp, NR / 2 warps a front, 32 / NR
// fronts at a time.
template <int NR, class T>
__device__ __noinline__ void fwd_warp_m(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I, FlowSlot &N,
                                        double *sm, uint32_t &wphase) {
  constexpr int WF = NR / 2, FR = 16 / WF, RT = kWarpSolveH / 32;
  const int     warp = threadIdx.x / 32, lane = threadIdx.x % 32, vg = 2 * (warp % WF);
  const long    polls = I.polls;
  double       *zs = sm + kFlowInvSmem + 128 * warp, *ys = zs + 64;
  panels_get(a, S, I, sm);
  flow_fetch(a, N);
  for (int q = warp / WF; q < I.item.nr; q += FR) {
    const FlowFront f = a.warps[I.item.r0 + q];
    const int       w = f.w, h = f.h, ld = h | 1;
    const double   *M = sm + f.part / 8 + lane;
    double          z[RT][2];
    FlowGather      g[RT];
    bool            more = false;
#pragma unroll
    for (int t = 0; t < RT; t++) {
      g[t] = FlowGather{kFlowNone, kFlowNone};
      if (lane + 32 * t < h) g[t] = a.gfirst[f.zofs + lane + 32 * t];
      z[t][0] = z[t][1] = 0.0;
      more |= g[t].more != kFlowNone;
    }
    if (lane < w) {
      z[0][0] = a.x[vg * a.n + f.col0 + lane];
      z[0][1] = a.x[(vg + 1) * a.n + f.col0 + lane];
    }
    // first children of all rows, polled together
    unsigned need = 0;
#pragma unroll
    for (int t = 0; t < RT; t++)
      if (g[t].first != kFlowNone) need |= 1u << t;
    for (long it = 0; need != 0; it++) {
      V2 raw[RT];
#pragma unroll
      for (int t = 0; t < RT; t++) {
        raw[t] = V2{kPending, kPending};
        if (need >> t & 1u) raw[t] = ld_relaxed_2(a.z + static_cast<int64_t>(NR) * g[t].first + vg);
      }
#pragma unroll
      for (int t = 0; t < RT; t++)
        if (raw[t].a != kPending && raw[t].b != kPending) {
          z[t][0] += __longlong_as_double(static_cast<long long>(raw[t].a));
          z[t][1] += __longlong_as_double(static_cast<long long>(raw[t].b));
          need &= ~(1u << t);
        }
      if (need != 0 && it >= polls) {
        atomicExch(a.err, 1);
        break;
      }
      if ((it & 63) == 63) {
        if (*reinterpret_cast<volatile int32_t *>(a.err) != 0) break;
        __nanosleep(32);
      }
    }
    if (more) {
#pragma unroll
      for (int t = 0; t < RT; t++)
        if (g[t].more != kFlowNone) {
          const uint32_t *m = a.gmore + g[t].more;
          for (uint32_t e = 1, n = m[0]; e <= n; e++)
            add_entry<2>(a.z + static_cast<int64_t>(NR) * m[e] + vg, true, z[t], a.err, polls);
        }
    }
    put_entry<2>(zs + 2 * lane, z[0]);
    __syncwarp();
    bulk_wait(smem_addr(&S.wbar[q]), wphase >> q & 1u, a.err);
    double y[2] = {0.0, 0.0};
#pragma unroll 4
    for (int k = 0; k < w; k++) fma_entry<2>(M[k * ld], zs + 2 * k, y);
    put_entry<2>(ys + 2 * lane, y);  // entries at or past w are not used
    __syncwarp();
    if (lane < w) {
      a.f[static_cast<int64_t>(NR) * (f.col0 + lane) + vg]     = y[0];
      a.f[static_cast<int64_t>(NR) * (f.col0 + lane) + vg + 1] = y[1];
    }
#pragma unroll
    for (int t = 0; t < RT; t++) {
      if (32 * t >= h) break;
      double u[2] = {0.0, 0.0};
#pragma unroll 4
      for (int k = 0; k < w; k++) fma_entry<2>(M[k * ld + 32 * t], ys + 2 * k, u);
      const int i = lane + 32 * t;
      if (i >= w && i < h && I.publish)
        st_relaxed_2(a.z + NR * (f.zofs + i) + vg, z[t][0] - u[0], z[t][1] - u[1]);
    }
    __syncwarp();
  }
  // Barrier q is used once an item, whichever warps wait on it.
  wphase ^= (1u << I.item.nr) - 1u;
}

template <int NR, class T>
__global__ void __launch_bounds__(kFlowThreads, 1) k_fwd_flow_m(const __grid_constant__ FlowArgs<T> a) {
  grid_wait();
  extern __shared__ __align__(128) double sm[];
  __shared__ __align__(16) FlowShared S;
  uint32_t phase = 0, wphase = 0;
  if (flow_idle(a)) return;
  flow_loop<true>(a, S, [&](const FlowSlot &I, FlowSlot &N) {
    switch (I.item.kind) {
      case kFlowWarps: fwd_warp_m<NR>(a, S, I, N, sm, wphase); break;
      case kFwdNarrow:
        if (I.item.f.w <= 32)
          fwd_narrow_m<16, NR>(a, S, I, N, sm, phase);
        else
          fwd_narrow_m<4, NR>(a, S, I, N, sm, phase);
        break;
      case kFwdSlab: fwd_slab_m<NR>(a, S, I, N, sm, phase); break;
      case kFwdSum: fwd_sum_m<NR>(a, I, N); break;
      default: fwd_rows_m<NR>(a, I, N, sm);
    }
  });
  flow_mark(a.mark, a.nmark);
}

// ---------------------------------------------------------------------------
// Backward.

// t(c, k) = sum_r L(r, c) x(r, k) over up to 512 rows below the block, for
// columns [c0, cend), at most 128: emit(c, k, t) by one lane a value.  ncg = 1,
// 2 or 4 groups of 32 columns by 16 / ncg groups of 32 ncg rows; the row groups
// are then added through out: at once (512 entries), or, where 16 vectors leave
// no room for that, pairwise (256 entries).
template <int NR, class T, class Emit>
__device__ __forceinline__ void chunk_cols_m(const FlowArgs<T> &a, const FlowFront &f, int64_t rb, int nr,
                                             int c0, int cend, double *xs, double *out, long polls,
                                             FlowSlot &N, Emit emit) {
  constexpr int NP  = kPitch<NR>;
  const int     tid = threadIdx.x, warp = tid / 32;
  const int     ncg = cend - c0 <= 32 ? 1 : cend - c0 <= 64 ? 2 : 4, cg = warp % ncg, rq = warp / ncg;
  const T      *P   = a.panel + f.panel;
  const int     c = c0 + 32 * cg, rw = 32 * ncg * rq;
  float         lv[32], lvn[32];
  load_frag_t(lv, P, f.h, rb + rw, rb + nr, c, cend);
  flow_fetch(a, N);
  const int row = tid < nr ? a.srows[f.rows + rb + tid] : -1;
  wait_gate(a, f.gate < 0 ? -1 : static_cast<int64_t>(NR) * f.gate, polls);
  get_entry<NR>(a.xr + static_cast<int64_t>(NR) * row, row >= 0, xs + NP * tid, a.err, polls);
  __syncthreads();
  Frag<NR> fr;
  fr.zero();
  for (int s = 0; s < ncg; s++) {
    if (s + 1 < ncg) load_frag_t(lvn, P, f.h, rb + rw + 32 * (s + 1), rb + nr, c, cend);
    mma_tile(fr, lv, xs + NP * (rw + 32 * s));
#pragma unroll
    for (int k = 0; k < 32; k++) lv[k] = lvn[k];
  }
  if (NR <= 8) {
    fr.template put<false>(out + NP * 32 * warp);
    __syncthreads();
    for (int e = tid; e < 32 * ncg * NR; e += kFlowThreads) {
      const int     col = c0 + e / NR;
      const double *q   = out + NP * (e / NR) + e % NR;
      double        t   = 0.0;
      for (int g = 0; g < 16 / ncg; g++) t += q[NP * 32 * ncg * g];
      if (col < cend) emit(col, e % NR, t);
    }
    return;
  }
  for (int half = 8 / ncg; half >= 1; half /= 2) {
    if (rq >= half && rq < 2 * half) fr.template put<false>(out + NP * 32 * (warp - half * ncg));
    __syncthreads();
    if (rq < half) fr.add(out + NP * 32 * warp);
    __syncthreads();
  }
  const int v = 2 * (threadIdx.x % 4);
  if (rq == 0 && (NR >= 8 || v < 4)) {
#pragma unroll
    for (int o = 0; o < 4; o++) {
      const int col = c + Frag<NR>::template row<false>(o);
#pragma unroll
      for (int n = 0; n < Frag<NR>::kN; n++)
        if (col < cend) {
          emit(col, 8 * n + v, fr.c[o][n][0]);
          emit(col, 8 * n + v + 1, fr.c[o][n][1]);
        }
    }
  }
}

template <int NR, class T>
__device__ __noinline__ void bwd_chunk_m(const FlowArgs<T> &a, const FlowSlot &I, FlowSlot &N, double *sm) {
  const FlowFront &f  = I.item.f;
  const int        c  = I.item.c0;
  const int64_t    rb = f.w + static_cast<int64_t>(c) * kFlowChunk;
  const int        nr = static_cast<int>(min(static_cast<int64_t>(kFlowChunk), f.h - rb));
  double          *pp = a.part + NR * (f.part + static_cast<int64_t>(c) * f.w);
  chunk_cols_m<NR>(a, f, rb, nr, I.item.r0, I.item.r0 + I.item.nr, sm + kFlowInvSmem, sm, I.polls, N,
                   [&](int col, int k, double t) { st_relaxed_f64(pp + NR * col + k, t); });
}

// The sum of the chunk partials of output e (column e / NR, vector e % NR),
// four polled at a time.
template <int NR, class T>
__device__ __forceinline__ double chunk_sum(const FlowArgs<T> &a, const FlowFront &f, int e, long polls) {
  const double *p = a.part + NR * f.part + e;
  const int64_t d = static_cast<int64_t>(NR) * f.w;
  double        s = 0.0;
  for (int c = 0; c < f.chunks; c += 4) {
    unsigned long long raw[4];
#pragma unroll
    for (int u = 0; u < 4; u++) raw[u] = c + u < f.chunks ? ld_relaxed_u64(p + (c + u) * d) : 0ull;
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (c + u < f.chunks) s += take_value(raw[u], p + (c + u) * d, a.err, polls);
  }
  return s;
}

template <int NR, class T>
__device__ __noinline__ void bwd_narrow_m(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I,
                                          FlowSlot &N, double *sm, uint32_t &phase) {
  const FlowFront &f   = I.item.f;
  const int        tid = threadIdx.x;
  const int        w = f.w, nbw = (w + 31) / 32;
  const long       polls = I.polls;
  constexpr int    KO = NR / 4, NP = kPitch<NR>;
  double          *inv = sm, *xs = sm + kNarrowInv, *vs = xs + 512 * kPitch<NR>, *out = vs + 128 * kPitch<NR>;
  const uint32_t   bar = smem_addr(&S.bar);
  if (tid == 0) {
    const uint32_t bytes = nbw * (nbw + 1) / 2 * kFlowBlk * sizeof(double);
    bulk_expect(bar, bytes);
    bulk_get(inv, a.inv + f.inv, bytes, bar);
  }
  // vs: the right-hand side less the rows below
  double v[KO];
#pragma unroll
  for (int m = 0; m < KO; m++) {
    const int e = tid + 512 * m;
    v[m]        = 0.0;
    if (e < w * NR) {
      v[m] = a.f[static_cast<int64_t>(NR) * f.col0 + e];
      if (a.Dinv) v[m] *= static_cast<double>(a.Dinv[f.col0 + e / NR]);
    }
  }
  if (f.chunks > 0 || f.h == w) flow_fetch(a, N);
  if (f.chunks == 0 && f.h > w) {
    chunk_cols_m<NR>(a, f, w, f.h - w, 0, w, xs, out, polls, N,
                     [&](int col, int k, double t) { vs[NP * col + k] = t; });
    __syncthreads();
  }
#pragma unroll
  for (int m = 0; m < KO; m++) {
    const int e = tid + 512 * m;
    if (e < w * NR && f.h > w) v[m] -= f.chunks > 0 ? chunk_sum<NR>(a, f, e, polls) : vs[NP * (e / NR) + e % NR];
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < KO; m++) {
    const int e = tid + 512 * m;
    if (e < 128 * NR) vs[NP * (e / NR) + e % NR] = v[m];
  }
  __syncthreads();
  bulk_wait(bar, phase, a.err);
  phase ^= 1;
  // x = Inv^T v: warp b takes the columns 32 b .., all blocks below
  const int b = tid / 32;
  if (b < nbw) {
    Frag<NR> fr;
    fr.zero();
    for (int i = b; i < nbw; i++)
      mma_inverse_t(fr, inv + (i * (i + 1) / 2 + b) * kFlowBlk, vs + 32 * NP * i);
    __syncwarp();
    fr.template put<false>(xs + 32 * NP * b);
  }
  __syncthreads();
#pragma unroll
  for (int m = 0; m < KO; m++) {
    const int e = tid + 512 * m;
    if (e < w * NR) {
      const double x = xs[NP * (e / NR) + e % NR];
      st_relaxed_f64(a.xr + static_cast<int64_t>(NR) * f.col0 + e, x);
      a.x[(e % NR) * a.n + f.col0 + e / NR] = x;
    }
  }
}

template <int NR, class T>
__device__ __noinline__ void bwd_slab_m(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I, FlowSlot &N,
                                        double *sm, uint32_t &phase) {
  const FlowFront &f   = I.item.f;
  const int        tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  constexpr int    NP  = kPitch<NR>;
  const int        col = tid / NR, vv = tid % NR, at = NP * col + vv;  // the thread's output, tid < 32 NR
  const long       polls = I.polls;
  const int        w = f.w, k0 = I.item.r0, s = k0 / kFlowSB, j = (k0 % kFlowSB) / 32;
  const int        nsl = min(16, (w - s * kFlowSB + 31) / 32), nsb = (w + kFlowSB - 1) / kFlowSB;
  const bool       mine = col < I.item.nr;
  double          *inv = sm, *xs = sm + kFlowInvSmem, *own = xs + 32 * NP * warp;
  const uint32_t   bar = smem_addr(&S.bar);
  if (tid == 0) {
    bulk_expect(bar, (nsl - j) * kFlowBlk * sizeof(double));
    for (int i = j; i < nsl; i++)
      bulk_get(inv + (i - j) * kFlowBlk,
               a.inv + f.inv +
                   (static_cast<int64_t>(s) * kFlowTriSB + i * (i + 1) / 2 + j) * kFlowBlk,
               kFlowBlk * sizeof(double), bar);
  }
  const T      *P    = a.panel + f.panel;
  const double *xr   = a.xr + ((I.ticket % kMultiCopies) * a.n + f.col0) * NR;
  const int     cend = k0 + I.item.nr;
  // Tile R: the warp takes the rows 32 warp .. of super-block R.
  const int64_t rw = 32 * warp;
  float         lv[32], lvn[32];
  if (nsb - 1 > s) load_frag_t(lv, P, f.h, (nsb - 1) * static_cast<int64_t>(kFlowSB) + rw, w, k0, cend);
  flow_fetch(a, N);
  double v = 0.0;
  if (mine) {
    v = a.f[static_cast<int64_t>(NR) * (f.col0 + k0) + tid];
    if (a.Dinv) v *= static_cast<double>(a.Dinv[f.col0 + k0 + col]);
    if (f.chunks > 0) v -= chunk_sum<NR>(a, f, NR * k0 + tid, polls);
  }
  Frag<NR> fr;
  fr.zero();
  for (int R = nsb - 1; R > s; R--) {
    const int64_t rb = R * static_cast<int64_t>(kFlowSB) + rw;
    if (R - 1 > s) load_frag_t(lvn, P, f.h, rb - kFlowSB, w, k0, cend);
    get_entry<NR>(xr + NR * (rb + lane), rb + lane < w, own + NP * lane, a.err, polls);
    __syncwarp();
    mma_tile(fr, lv, own);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 32; k++) lv[k] = lvn[k];
  }
  if (nsb - 1 > s) {
    fr.template put<false>(own);
    __syncthreads();
    if (col < 32) {
      double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int q = 0; q < 16; q++) t[q % 4] += xs[32 * NP * q + at];
      v -= (t[0] + t[1]) + (t[2] + t[3]);
    }
    __syncthreads();
  }
  double *xz = a.xz + static_cast<int64_t>(NR) * (f.col0 + s * kFlowSB);
  if (col < 32) {
    if (!mine) v = 0.0;
    if (j > 0 && mine) st_relaxed_f64(xz + 32 * NR * j + tid, v);
    xs[at] = v;  // the diagonal block's, for warp 0
  }
  __syncthreads();
  bulk_wait(bar, phase, a.err);
  phase ^= 1;
  if (j + warp < nsl) {
    const int i = j + warp;
    if (warp > 0)
      get_entry<NR>(xz + NR * (32 * i + lane), s * kFlowSB + 32 * i + lane < w, own + NP * lane, a.err,
                    polls);
    __syncwarp();
    fr.zero();
    mma_inverse_t(fr, inv + warp * kFlowBlk, own);
    __syncwarp();
    fr.template put<false>(own);
  }
  __syncthreads();
  if (mine) {
    double t[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 16; q++)
      if (j + q < nsl) t[q % 4] += xs[32 * NP * q + at];
    const double  x = (t[0] + t[1]) + (t[2] + t[3]);
    const int64_t g = static_cast<int64_t>(NR) * (f.col0 + k0) + tid;
#pragma unroll
    for (int c = 0; c < kMultiCopies; c++) st_relaxed_f64(a.xr + c * a.n * NR + g, x);
    a.x[vv * a.n + f.col0 + k0 + col] = x;
  }
}

template <int NR, class T>
__device__ __noinline__ void bwd_warp_m(const FlowArgs<T> &a, FlowShared &S, const FlowSlot &I, FlowSlot &N,
                                        double *sm, uint32_t &wphase) {
  constexpr int WF = NR / 2, FR = 16 / WF, RT = kWarpSolveH / 32;
  const int     warp = threadIdx.x / 32, lane = threadIdx.x % 32, vg = 2 * (warp % WF);
  const long    polls = I.polls;
  double       *vs = sm + kFlowInvSmem + 576 * warp, *xs = vs + 64;
  panels_get(a, S, I, sm);
  flow_fetch(a, N);
  for (int q = warp / WF; q < I.item.nr; q += FR) {
    const FlowFront f = a.warps[I.item.r0 + q];
    const int       w = f.w, h = f.h, ld = h | 1, nr = h - w;
    double          v[2] = {0.0, 0.0};
    if (lane < w) {
      const double *p = a.f + static_cast<int64_t>(NR) * (f.col0 + lane) + vg;
      const double  d = a.Dinv ? static_cast<double>(a.Dinv[f.col0 + lane]) : 1.0;
      v[0]            = p[0] * d;
      v[1]            = p[1] * d;
    }
    {
      int    gi[RT];
      double xv[RT][2];
#pragma unroll
      for (int t = 0; t < RT; t++) {
        gi[t]    = lane + 32 * t < nr ? a.srows[f.rows + w + lane + 32 * t] : -1;
        xv[t][0] = xv[t][1] = 0.0;
      }
      wait_gate(a, f.gate < 0 ? -1 : static_cast<int64_t>(NR) * f.gate, polls);
      unsigned need = 0;
#pragma unroll
      for (int t = 0; t < RT; t++)
        if (gi[t] >= 0) need |= 1u << t;
      for (long it = 0; need != 0; it++) {
        V2 raw[RT];
#pragma unroll
        for (int t = 0; t < RT; t++) {
          raw[t] = V2{kPending, kPending};
          if (need >> t & 1u) raw[t] = ld_relaxed_2(a.xr + static_cast<int64_t>(NR) * gi[t] + vg);
        }
#pragma unroll
        for (int t = 0; t < RT; t++)
          if (raw[t].a != kPending && raw[t].b != kPending) {
            xv[t][0] = __longlong_as_double(static_cast<long long>(raw[t].a));
            xv[t][1] = __longlong_as_double(static_cast<long long>(raw[t].b));
            need &= ~(1u << t);
          }
        if (need != 0 && it >= polls) {
          atomicExch(a.err, 1);
          break;
        }
        if ((it & 63) == 63) {
          if (*reinterpret_cast<volatile int32_t *>(a.err) != 0) break;
          __nanosleep(32);
        }
      }
#pragma unroll
      for (int t = 0; t < RT; t++) put_entry<2>(xs + 2 * (lane + 32 * t), xv[t]);
    }
    __syncwarp();
    bulk_wait(smem_addr(&S.wbar[q]), wphase >> q & 1u, a.err);
    const bool    half = w <= 16;
    const double *col  = sm + f.part / 8 + min(half ? lane & 15 : lane, w - 1) * ld;
    const int     step = half ? 2 : 1;
    double        t[2] = {0.0, 0.0};
#pragma unroll 4
    for (int r = half ? lane >> 4 : 0; r < nr; r += step) fma_entry<2>(col[w + r], xs + 2 * r, t);
    if (half) {
      t[0] += __shfl_xor_sync(0xffffffffu, t[0], 16);
      t[1] += __shfl_xor_sync(0xffffffffu, t[1], 16);
    }
    v[0] = lane < w ? v[0] - t[0] : 0.0;
    v[1] = lane < w ? v[1] - t[1] : 0.0;
    put_entry<2>(vs + 2 * lane, v);
    __syncwarp();
    double x[2] = {0.0, 0.0};
#pragma unroll 4
    for (int i = 0; i < w; i++) fma_entry<2>(col[i], vs + 2 * i, x);
    if (lane < w) {
      st_relaxed_2(a.xr + static_cast<int64_t>(NR) * (f.col0 + lane) + vg, x[0], x[1]);
      a.x[vg * a.n + f.col0 + lane]       = x[0];
      a.x[(vg + 1) * a.n + f.col0 + lane] = x[1];
    }
    __syncwarp();
  }
  wphase ^= (1u << I.item.nr) - 1u;
}

template <int NR, class T>
__global__ void __launch_bounds__(kFlowThreads, 1) k_bwd_flow_m(const __grid_constant__ FlowArgs<T> a) {
  grid_wait();
  extern __shared__ __align__(128) double sm[];
  __shared__ __align__(16) FlowShared S;
  uint32_t phase = 0, wphase = 0;
  if (flow_idle(a)) return;
  flow_loop<true>(a, S, [&](const FlowSlot &I, FlowSlot &N) {
    switch (I.item.kind) {
      case kFlowWarps: bwd_warp_m<NR>(a, S, I, N, sm, wphase); break;
      case kBwdChunk: bwd_chunk_m<NR>(a, I, N, sm); break;
      case kBwdNarrow: bwd_narrow_m<NR>(a, S, I, N, sm, phase); break;
      default: bwd_slab_m<NR>(a, S, I, N, sm, phase);
    }
  });
  flow_mark(a.mark, a.nmark);
}

// The handed-over values in one buffer, in entries of NR values.
struct MultiBuffers {
  int64_t fwd, bwd;
  explicit MultiBuffers(const Plan &P)
      : fwd(P.flow_z_elems + (kMultiCopies + 1) * P.S.n),
        bwd(P.flow_part_elems + (kMultiCopies + 1) * P.S.n) {}
};

template <int NR, class T>
void solve_multi_nr(const Plan &P, const Numeric &F, const T *pan, double *X,
                    MultiSolveWorkspace &ws, cudaStream_t s, const ActiveFlags &act) {
  const int64_t      n = P.S.n;
  KernelTimer       &kt = kernel_timer();
  const MultiBuffers b(P);
  double            *fv = ws.vals.as<double>(), *bv = fv + NR * b.fwd;
  FlowArgs<T>        a{};
  a.warps  = P.flow_warp.as<FlowFront>();
  a.panel  = pan;
  a.inv    = F.inv64.as<double>();
  a.wpanel = F.wpanel.as<double>();
  a.gfirst = P.flow_gfirst.as<FlowGather>();
  a.gmore  = P.flow_gmore.as<uint32_t>();
  a.srows  = P.srows.as<int32_t>();
  a.n      = n;
  a.x      = X;
  a.f      = bv + NR * b.bwd;
  a.z      = fv;
  a.y      = a.z + NR * P.flow_z_elems;
  a.yz     = a.y + NR * kMultiCopies * n;
  a.part   = bv;
  a.xr     = a.part + NR * P.flow_part_elems;
  a.xz     = a.xr + NR * kMultiCopies * n;
  a.err    = ws.err.as<int32_t>();
  a.active        = act.p;
  a.nactive       = act.count;
  a.active_stride = act.stride;
  constexpr int smem = kMultiSmem * sizeof(double);
  kt.begin(kKcSolveFwd, s);
  if (!ws.fwd_pending) flow_pending(fv, NR * b.fwd, s);
  a.items  = P.flow_fwd.as<FlowItem>();
  a.nitems = P.nflow_fwd;
  a.mark   = bv;
  a.nmark  = NR * b.bwd;
  a.ticket = ws.sync.as<int32_t>();
  launch_chained(n, k_fwd_flow_m<NR, T>, 1, std::min(P.nflow_fwd, kSMs), kFlowThreads, smem, s, a);
  kt.end(s);
  MPIR_CHECK_LAUNCH();
  kt.begin(kKcSolveBwd, s);
  a.items  = P.flow_bwd.as<FlowItem>();
  a.nitems = P.nflow_bwd;
  a.mark   = fv;
  a.nmark  = NR * b.fwd;
  a.Dinv   = F.Dinv.as<float>();
  a.ticket = ws.sync.as<int32_t>() + 1;
  launch_chained(n, k_bwd_flow_m<NR, T>, 1, std::min(P.nflow_bwd, kSMs), kFlowThreads, smem, s, a);
  ws.fwd_pending = true;
  kt.end(s);
  MPIR_CHECK_LAUNCH();
}

template <int NR>
void allow_multi() {
  static OncePerDevice attr;
  allow_smem(attr, kMultiSmem * sizeof(double),
             {reinterpret_cast<const void *>(k_fwd_flow_m<NR, float>), reinterpret_cast<const void *>(k_bwd_flow_m<NR, float>),
              reinterpret_cast<const void *>(k_fwd_flow_m<NR, __half>),
              reinterpret_cast<const void *>(k_bwd_flow_m<NR, __half>),
              reinterpret_cast<const void *>(k_fwd_flow_m<NR, __nv_bfloat16>),
              reinterpret_cast<const void *>(k_bwd_flow_m<NR, __nv_bfloat16>)});
}

}  // namespace

int multi_width(int nrhs) {
  if (nrhs <= 4) return 4;
  if (nrhs <= 8) return 8;
  return 16;
}

void MultiSolveWorkspace::allocate(const Plan &P, int width) {
  const MultiBuffers b(P);
  nr          = 0;  // until all of it is there
  fwd_pending = false;
  vals.resize(std::max<int64_t>((b.fwd + b.bwd + P.S.n) * width, 1) * sizeof(double));
  sync.resize(4 * sizeof(int32_t));
  device_zero(sync.as<void>(), sync.bytes());
  err.resize(sizeof(SolveCtl));
  device_zero(err.as<void>(), sizeof(SolveCtl));
  if (width == 4) allow_multi<4>();
  if (width == 8) allow_multi<8>();
  if (width == 16) allow_multi<16>();
  nr = width;
}

size_t MultiSolveWorkspace::bytes_for(const Plan &P, int width) {
  const MultiBuffers b(P);
  return (b.fwd + b.bwd + P.S.n) * width * sizeof(double) + 4 * sizeof(int32_t) + sizeof(SolveCtl);
}

void ldlt_solve_multi(const Plan &P, const Numeric &F, double *X, int width,
                      MultiSolveWorkspace &ws, cudaStream_t s, const ActiveFlags &act) {
  if (P.S.n == 0) return;
  if (ws.nr != width) throw std::logic_error("multi-vector workspace of another width");
  if (width != 4 && width != 8 && width != 16)
    throw std::invalid_argument("multi-vector solve width must be 4, 8 or 16");
  auto run = [&](auto *pan) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(pan)>>;
    if (width == 4) solve_multi_nr<4, T>(P, F, pan, X, ws, s, act);
    if (width == 8) solve_multi_nr<8, T>(P, F, pan, X, ws, s, act);
    if (width == 16) solve_multi_nr<16, T>(P, F, pan, X, ws, s, act);
  };
  switch (F.solve_prec()) {
    case 2: run(F.panel16.as<const __nv_bfloat16>()); break;
    case 3: run(F.panel16.as<const __half>()); break;
    default: run(F.panel.as<const float>());
  }
}

}  // namespace mpir
