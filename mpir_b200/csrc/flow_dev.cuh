// Device code shared by the dataflow triangular solves for one vector (solve.cu)
// and for several (solve_multi.cu): the work-item loop, the hand-over of
// values and the loads of L.
#pragma once
#include "common.cuh"
#include "flow.cuh"
#include "solve_dev.cuh"

namespace mpir {

constexpr int kFlowThreads = 512;
constexpr int kFlowCopies  = 4;  // copies of a wide front's block results

// Shared memory of the kernels (doubles): the staged inverse blocks (or the
// panels of the warp-solved fronts), then vectors and partial sums.
constexpr int kFlowInvSmem = 16 * kFlowBlk;
static_assert(kFlowInvSmem * 8 == kFlowPanelSmem, "the host packs panels into the same space");

template <class T>
struct FlowArgs {
  const FlowItem  *items;
  int32_t          nitems;
  const FlowFront *warps;
  const T         *panel;
  const double    *inv, *wpanel;
  const FlowGather *gfirst;
  const uint32_t   *gmore;
  const int32_t   *srows;
  const float     *Dinv;  // backward: f .* Dinv is its right-hand side (NULL: f)
  int64_t          n;
  // Forward: x in, f out (several items of a front read its entries of x).
  // Backward: f in, x out.
  double          *x, *f;
  // Values handed over: forward z (children's update vectors), y (block
  // results, kFlowCopies x n), yz (right-hand sides inside a super-block);
  // backward xr (results, kFlowCopies x n), xz, part (chunk partials).
  double  *z, *y, *yz, *xr, *xz, *part;
  double  *mark;    // the other direction's values, marked pending at the end
  int64_t  nmark;
  int32_t *ticket;
  int32_t *err;
  // nactive flags active_stride apart (NULL: none): nothing is done when all
  // are zero (the values stay as they are, for the next solve).
  const int32_t *active;
  int32_t        nactive;
  int64_t        active_stride;
};

struct FlowSlot {
  FlowItem item;
  int32_t  ticket;
  int32_t  publish;
  long     polls;
};
struct FlowShared {
  FlowSlot slot[2];
  uint64_t bar;                       // inverse blocks
  uint64_t wbar[kFlowWarpsPerItem];   // a warp's panel
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// The CTA's next ticket and its item, by the last warp (the last CTA to find
// none resets the counter for the next launch).  Called by each item's work
// once its first loads are on their way, one item ahead: the two round trips
// (ticket, item) are then off the path between items.  A CTA so holds at most
// one ticket beyond the item it works on, and the lowest ticket not done is
// always being worked on.
template <class T>
__device__ __forceinline__ void flow_fetch(const FlowArgs<T> &a, FlowSlot &S) {
  if (threadIdx.x < kFlowThreads - 32) return;
  const int lane = threadIdx.x % 32;
  int       t    = 0;
  if (lane == 0) {
    t = atomicAdd(a.ticket, 1);
    if (t == a.nitems + static_cast<int>(gridDim.x) - 1) *a.ticket = 0;
    const volatile SolveCtl *c = reinterpret_cast<const volatile SolveCtl *>(a.err);
    S.ticket  = t;
    S.polls   = poll_limit(c->poll_log2);
    S.publish = c->withhold != t + 1;
  }
  t = __shfl_sync(0xffffffffu, t, 0);
  if (t < a.nitems && lane < kFlowItemWords)
    cp_async8(reinterpret_cast<double *>(&S.item) + lane,
              reinterpret_cast<const double *>(a.items + t) + lane);
}

// True when no vector is active: the kernel returns at once (no ticket taken,
// no value marked).
template <class T>
__device__ __forceinline__ bool flow_idle(const FlowArgs<T> &a) {
  int32_t on = a.active == nullptr;
  for (int k = 0; k < a.nactive; k++) on |= a.active[k * a.active_stride];
  return on == 0;
}

// The kernels' common loop: work(this slot, the next one) for every item.
// kStores: an item's ordinary stores may lie where the next one's bulk copies
// go.  Those copies are of the async proxy, which a barrier alone does not
// order after the stores.
template <bool kStores, class T, class Work>
__device__ __forceinline__ void flow_loop(const FlowArgs<T> &a, FlowShared &S, Work work) {
  if (threadIdx.x <= kFlowWarpsPerItem) {
    const uint32_t b = smem_addr(threadIdx.x == 0 ? &S.bar : &S.wbar[threadIdx.x - 1]);
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  flow_fetch(a, S.slot[0]);
  cp_async_wait_all();
  __syncthreads();
  for (int k = 0; S.slot[k & 1].ticket < a.nitems; k++) {
    work(S.slot[k & 1], S.slot[(k + 1) & 1]);
    cp_async_wait_all();
    if (kStores) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
  }
}

// Bulk copies of inverse blocks into shared memory, completing on S.bar.
__device__ __forceinline__ void bulk_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_get(double *dst, const double *src, uint32_t bytes,
                                         uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void bulk_wait(uint32_t bar, uint32_t parity, int32_t *err) {
  for (long it = 0; it < 20000000; it++) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred P1;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, P1;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return;
  }
  atomicExch(err, 1);
}

// The value at p from a load issued ahead (raw) when that load already saw
// it, else the wait for it.
__device__ __forceinline__ double take_value(unsigned long long raw, const double *p,
                                             int32_t *err, long polls) {
  return raw != kPending ? __longlong_as_double(static_cast<long long>(raw))
                         : wait_value(p, err, polls);
}

// A row's child contributions, in child order: the first one's index sits
// with the row, the others (few rows have any) in a list after their count.
// begin() issues the loads of the index and the first value, finish() waits
// for what is pending and adds the rest, four at a time.  Entry i's values of
// NR vectors are at NR i; z points at the vector's own of entry 0.
template <int NR>
struct Gather {
  FlowGather         g = {kFlowNone, kFlowNone};
  unsigned long long r0 = 0;
  template <class T>
  __device__ __forceinline__ void begin(const FlowArgs<T> &a, int64_t row, const double *z) {
    g = a.gfirst[row];
    if (g.first != kFlowNone) r0 = ld_relaxed_u64(z + static_cast<int64_t>(NR) * g.first);
  }
  template <class T>
  __device__ __forceinline__ double finish(const FlowArgs<T> &a, const double *z, double zr,
                                           long polls) {
    if (g.first != kFlowNone)
      zr += take_value(r0, z + static_cast<int64_t>(NR) * g.first, a.err, polls);
    if (g.more == kFlowNone) return zr;
    const uint32_t *m = a.gmore + g.more + 1;
    const uint32_t  n = m[-1];
    for (uint32_t q = 0; q < n; q += 4) {
      uint32_t           idx[4];
      unsigned long long raw[4];
#pragma unroll
      for (int u = 0; u < 4; u++) idx[u] = q + u < n ? m[q + u] : kFlowNone;
#pragma unroll
      for (int u = 0; u < 4; u++)
        raw[u] = idx[u] != kFlowNone ? ld_relaxed_u64(z + static_cast<int64_t>(NR) * idx[u]) : 0ull;
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (idx[u] != kFlowNone)
          zr += take_value(raw[u], z + static_cast<int64_t>(NR) * idx[u], a.err, polls);
    }
    return zr;
  }
};

// z[t] += the value at v + ix[t] (kFlowNone: none), all of them polled together.
template <int K>
__device__ __forceinline__ void add_values(const double *v, const uint32_t (&ix)[K], double (&z)[K],
                                           int32_t *err, long polls) {
  unsigned need = 0;
#pragma unroll
  for (int t = 0; t < K; t++)
    if (ix[t] != kFlowNone) need |= 1u << t;
  for (long it = 0; need != 0; it++) {
    unsigned long long raw[K];
#pragma unroll
    for (int t = 0; t < K; t++) raw[t] = (need >> t & 1u) ? ld_relaxed_u64(v + ix[t]) : kPending;
#pragma unroll
    for (int t = 0; t < K; t++)
      if (raw[t] != kPending) {
        z[t] += __longlong_as_double(static_cast<long long>(raw[t]));
        need &= ~(1u << t);
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

// Marks the other direction's values pending, the CTA's share of them.
__device__ __forceinline__ void flow_mark(double *p, int64_t n) {
  unsigned long long *q = reinterpret_cast<unsigned long long *>(p);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    q[i] = kPending;
}

// L(r, c0 + k) for k < 32, zero at or past column cend or when !rok.
template <class T>
__device__ __forceinline__ void load_cols(float (&d)[32], const T *P, int64_t h, int64_t r,
                                          bool rok, int c0, int cend) {
  const T  *p  = P + r + static_cast<int64_t>(c0) * h;
  const int nc = rok ? cend - c0 : 0;
#pragma unroll
  for (int k = 0; k < 32; k++) d[k] = k < nc ? to_f(__ldg(p + k * h)) : 0.0f;
}

// Rows rb + lane + 32 i (i < 16, nr valid) of columns c0 + 2 v, c0 + 2 v + 1
// (v = the warp, below cend).
template <class T>
__device__ __forceinline__ void load_rows(float (&d)[2][16], const T *P, int64_t h, int64_t rb,
                                          int nr, int c0, int cend) {
  const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
#pragma unroll
  for (int j = 0; j < 2; j++) {
    const int c = c0 + 2 * warp + j;
    const T  *p = P + rb + lane + static_cast<int64_t>(c) * h;
#pragma unroll
    for (int i = 0; i < 16; i++)
      d[j][i] = (c < cend && lane + 32 * i < nr) ? to_f(__ldg(p + 32 * i)) : 0.0f;
  }
}

// Backward items are taken long before the x they wait on are there, up to
// 512 of them a CTA.  Until the front's gate is ready one lane a warp polls
// that alone: all lanes polling their own entries from the start took enough
// of L2 to triple the time of a level (n = 1,280: 12 to 16 us a level).
template <class T>
__device__ __forceinline__ void wait_gate(const FlowArgs<T> &a, int64_t gate, long polls) {
  if (gate >= 0 && threadIdx.x % 32 == 0) wait_value(a.xr + gate, a.err, polls);
  __syncwarp();
}

// The float64 panel of a warp-solved front (k_flow_wpanel) into its place in
// shared memory, one bulk copy.
template <class T>
__device__ __forceinline__ const double *warp_panel(const FlowArgs<T> &a, const FlowFront &f,
                                                    double *sm, uint32_t bar) {
  double *dst = reinterpret_cast<double *>(reinterpret_cast<char *>(sm) + f.part);
  if (threadIdx.x % 32 == 0) {
    const uint32_t bytes = flow_wpanel_elems(f.w, f.h) * sizeof(double);
    bulk_expect(bar, bytes);
    bulk_get(dst, a.wpanel + f.inv, bytes, bar);
  }
  return dst;
}

}  // namespace mpir
