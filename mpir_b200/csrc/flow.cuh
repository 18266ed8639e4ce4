// Tables and device helpers of the dataflow triangular solves (solve.cu).
#pragma once
#include <cstdint>
#include <stdexcept>

namespace mpir {

// Entries of the front vectors are numbered in 32 bits without a sign (half of
// what 64 would have a row's gather read); kFlowNone is no entry.  2^32 of them
// do not fit the device: an entry takes 24 bytes in the front vectors, FlowGather
// and the row indices and 12 a column in the float32 and float64 panels, and a
// front has two columns (merged with its last child, at least) or is a leaf, whose
// entries are the matrix's, at 88 bytes each: 206 GB of 192.
constexpr uint32_t kFlowNone = 0xffffffffu;
inline uint32_t    flow_entry(int64_t i) {
  if (i < 0 || i >= static_cast<int64_t>(kFlowNone))
    throw std::invalid_argument("front vectors of more than 2^32 entries");
  return static_cast<uint32_t>(i);
}
// A row's child contributions: the first one's entry, and where the others lie
// in the list of further ones (their number, then their entries).  A row with
// more than kFlowFan (a star's centre has one for each of its points) has sums of
// kFlowFan of them instead, or sums of such sums, at most 8: entries behind the
// front vectors, formed by kFwdSum items.
constexpr int kFlowFan = 32;
struct alignas(8) FlowGather {
  uint32_t first, more;
};

// One front in the triangular solves.
struct FlowFront {
  int64_t panel;   // panel offset (h x w, column-major)
  int64_t zofs;    // front vector in the solve workspace (h entries); row i's
                   // child contributions start at gfirst[zofs + i]
  int64_t inv;     // float64 inverse of the diagonal block; of a warp-solved
                   // front: its float64 panel
  int64_t part;    // backward chunk partials (chunks x w doubles); of a
                   // warp-solved front: its panel's byte in shared memory
  int64_t rows;    // the front's row index set at srows[rows ..]
  int32_t h, w;
  int32_t col0;    // permuted index of the front's first column
  int32_t chunks;  // backward chunk items per column
  int32_t gate;    // backward: a column whose x is ready before the last x that
                   // the front waits on, and hardly before (-1: none)
  int32_t pad;
};

// One work item: a copy of its front's descriptor, the kind, and a range.
struct FlowItem {
  FlowFront f;
  int32_t   kind;
  int32_t   r0;  // first row (forward) or column (backward); kWarps: first entry
  int32_t   nr;  // rows or columns; kWarps: number of fronts
  int32_t   c0;  // kBwdChunk: chunk index
};
constexpr int kFlowItemWords = sizeof(FlowItem) / 8;
static_assert(sizeof(FlowItem) == 80, "copied in 8-byte words");

enum FlowKind : int32_t {
  kFlowWarps = 0,     // up to 16 fronts of the warp list, one warp each
  kFwdNarrow,         // w <= kFlowNarrow: the block solve and up to 512 of the
                      // rows below it
  kFwdSlab,           // w > kFlowNarrow: 32 rows of the diagonal block
  kFwdRows,           // w > kFlowNarrow: 128 rows below the diagonal block
  kFwdSum,            // nr <= 32 sums of kFlowFan contributions each, at zofs ..;
                      // their sources lie one after another from gmore[rows] on
  kBwdChunk,          // up to 512 rows below the block x up to 128 columns
  kBwdNarrow,         // w <= kFlowNarrow: the whole diagonal block
  kBwdSlab,           // w > kFlowNarrow: 32 columns of the diagonal block
};

// The inverse of a front's unit-lower diagonal block is kept per super-block
// of 512 columns, as 32 x 32 blocks of its lower block triangle: block (i, j),
// j <= i, of super-block s at (136 s + i (i + 1) / 2 + j) * kFlowBlk, entry
// (r, c) at c * 33 + r (the odd pitch makes reads along rows and along
// columns free of bank conflicts).
constexpr int kFlowSB     = 512;
constexpr int kFlowBlk    = 33 * 32;
constexpr int kFlowNarrow = 128;
constexpr int kFlowTriSB  = 16 * 17 / 2;
constexpr int kFlowRows   = 512;  // rows of a kFwdNarrow item, at most
constexpr int kFlowRowsW  = 128;  // rows of a kFwdRows item
constexpr int kFlowChunk  = 512;  // rows of a kBwdChunk item
constexpr int kFlowChunkC = 128;  // columns of one
constexpr int kFlowWarpsPerItem = 16;
// From this many items of leaves of at most 64 rows on, the solves for one
// vector take them by kernels of their own (k_fwd_leaf, k_bwd_leaf).
constexpr int kFlowLeafItems = 6 * 148;
constexpr int kFlowPanelSmem = 16 * kFlowBlk * 8;  // bytes for a kFlowWarps item's panels

// Doubles of a warp-solved front's float64 panel (even: copied in 16-byte words).
__host__ __device__ constexpr int flow_wpanel_elems(int w, int h) {
  return ((h | 1) * w + 1) / 2 * 2;
}

// Blocks of the inverse of a w-column front.
constexpr int64_t flow_inv_blocks(int64_t w) {
  const int64_t full = w / kFlowSB, b = (w % kFlowSB + 31) / 32;
  return full * kFlowTriSB + b * (b + 1) / 2;
}

// Strip of 16 columns of one super-block's inverse (k_flow_invert).
struct FlowInvDesc {
  int64_t panel;  // panel offset of the super-block's (0, 0)
  int64_t inv;    // its inverse (doubles)
  int32_t h;      // panel leading dimension
  int32_t n;      // columns of the super-block
  int32_t c0;     // first column of the strip
  int32_t pad;
};

}  // namespace mpir
