// Tensor-core products of the HODLR operator for 64 right-hand sides at once
// (tcgen05.cu).
//
// Vectors are "point major": entry p of a 64-column block sits at
// v[p * 64 .. p * 64 + 63], for the inputs [x | z] (tree positions, then the
// z values of the low-rank blocks) and for the FP32 output slots.  Inputs are
// stored split once: each value as a packed pair of BF16 words, the high part
// in the low half-word and the rest in the high half-word (x = hi + lo to
// about 2^-17 relative).  Each product is D (128 x N) = A (128 x K) B^T on the
// tensor cores: A holds the 64 right-hand sides' high parts (rows 0-63) and
// low parts (rows 64-127), B the factor columns (N output rows, K input
// columns in steps of 32), D the FP32 accumulator in tensor memory; the
// result is D_hi + D_lo.  BF16 factors times their input scale (BF16 dense
// tiles) are split into two BF16 terms, FP64 near-field entries into three
// (about 2^-24 relative).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "matvec.h"

namespace hodlr {

constexpr int kTcRhs = 64;     // right-hand sides per block
constexpr int kTcMaxSegs = 256;  // segments of one panel item (the host splits longer items)
// Output rows of one item: panels above 32 rows go in items of 64 rows, and z
// groups hold at most 64 rows -- so a CTA holds at most 64 tensor-memory
// columns and 8 CTAs share an SM.  Split items' partial sums are blocks of
// kTcRows rows.
constexpr int kTcRows = 64;

// kind of product: z = V^T x, near-field panels (FP64 tiles), far-field panels
// (BF16 dense tiles and U factors).  Panels of at most 32 rows, their low-rank
// blocks included, take the kernel of tcleaf.cu instead where the plan's rule says
// that it pays (build_tc_plan).
enum TcKind { kTcZ = 0, kTcNear = 1, kTcFar = 2 };

// z = V^T x for the low-rank blocks with one source node, grouped: the
// group's rows are rows k0 .. k0 + nk - 1 of z_b for each of its entries
// (at most kTcRows rows in all), and its columns the source node's points.
struct TcZEntry {
  int32_t zb;      // index into the z blocks
  int32_t k0, nk;  // rows (columns of V) of z_b in this group
};
struct TcZGroup {
  int64_t x_off;   // first point of the group's columns (of the source node)
  int32_t n;       // columns: all points of the source node, or a run of about kTcZCols of them
  int32_t e_begin, e_end;  // entries
  int32_t rows;    // sum of nk
  int32_t part;    // < 0: the group writes z; else its partial sums go to part block `part` (a fix-up adds them)
  int32_t col0;    // the first column's point within the source node (its row of V): 0 unless a column run
};
// A source node with more points than about kTcZCols is split into column runs
// whose partial sums (blocks of kTcRows rows x 64) a fix-up adds into z.  A CTA
// works through its run step by step, so long runs leave SMs idle (runs of 512
// instead of 256: 3D N = 30000 725 -> 874 us, 2D N = 18000 159 -> 176); but a node just
// above the limit is not worth two (4D N = 65536, whose leaves' parents have 256
// points on average: half of them split took 3.94 ms, none 3.55).
constexpr int kTcZCols = 256;
struct TcZRow {        // row i of a split group: where its z goes
  int64_t zpos;
  const float* zscale;  // the row's z scale (BF16), or null
};
struct TcZFix {
  int32_t part, count;  // part blocks part .. part + count - 1
  int32_t rows, row0;   // rows, and their first entry in the TcZRow table
};

struct TcLaunch {
  uint32_t* in;     // [x | z], point major, packed BF16 pairs
  float* y;         // output slots, point major: slot s of row p at (s * n + p) * 64
  float* part;      // partial row blocks of split panels: (part * rows_per_item + i) * 64
  int64_t n;        // points (rows of one slot)
  unsigned int* status;  // wait give-ups
  // panels (near, far)
  const Panel* panels;
  const Seg* segs;
  const Item* items;
  int nitems;       // 64-row chunks of panels above 32 rows
  // z products: blocks, groups by source node, group entries
  const ZBlock* zb;
  const TcZGroup* zgroups;
  const TcZEntry* zentries;
  int nz;           // groups
  int nmax;         // largest output row count of the launch's items (N before padding)
};

// ---- leaf-level products (tcleaf.cu): panels of at most 32 rows ----
// One segment of such a panel: a near tile (FP64) or a dense far tile (BF16,
// scale: its column scales), columns = the source's n points; or a low-rank
// block (V non-null): U m x K, V n x vstride row major, scale: z's K scales.
struct alignas(16) TcLeafSeg {
  const void* A;
  const uint16_t* V;
  const float* scale;
  int32_t n;
  int32_t K;
  int32_t vstride;
  int32_t unit;  // its source's first unit within the batch
};
// 8 points of a source (n < 8 in its last unit): one operand fragment set
struct TcUnit {
  int64_t x_off;
  int32_t n, pad;
};
constexpr int kTcUnitBytes = 2048;  // 64 right-hand sides x 8 points, high and low parts
constexpr uint64_t kTcWaitNs = 2000000000ull;  // the longest wait of a leaf-level kernel for a stage
constexpr int kTcLeafGroup = 8;     // panels of a group: one per warp of a CTA
// a batch of sources: at most kTcLeafUnits units, kTcLeafSegs segments and 32
// sources (two stages of 45 KB, two CTAs per SM)
constexpr int kTcLeafUnits = 20;
constexpr int kTcLeafSegs = 96;
struct TcLeafSrc {
  int32_t xunit, n;  // first unit; points (at most 8 kTcLeafUnits)
};
struct alignas(16) TcLeafBatch {
  int32_t src_b, src_e;
  int32_t seg_b;                       // its segments, by panel of the group:
  int32_t warp_off[kTcLeafGroup + 1];  // panel w's are seg_b + warp_off[w] .. warp_off[w + 1] - 1
};
// A group's run of batches: panels panel0 .. panel0 + count - 1 of the near or
// far list; part < 0: the outputs, else panel w's partial block part + w * part_stride.
struct TcLeafRun {
  int32_t near, panel0, count;
  int32_t batch_b, batch_e;
  int32_t part, part_stride;
};
struct TcLeafArgs {
  const Panel *near_panels, *far_panels;
  const int32_t *near_list, *far_list;  // the panels of at most 32 rows
  const TcLeafSeg *near_segs, *far_segs;  // in batch order
  const TcLeafSrc* srcs;
  const TcLeafBatch* batches;
  const TcLeafRun* runs;
  int nruns;
  const uint4* xunits;  // 128 per unit
  float* y;
  float *part_near, *part_far;  // part blocks of kTcRows x 64
  unsigned int* status;  // counts the warps that gave up a wait (the results are invalid then)
  uint64_t wait_ns;      // the longest wait for a stage
  // tests only: the batch of each run whose copies are left out, and the one
  // after which warp 1 does not hand its stage back (-1: none)
  int32_t drop_copies, drop_release;
};
cudaError_t launch_tc_units(const uint32_t* in, const TcUnit* units, int64_t nunits, uint4* out, cudaStream_t st);
cudaError_t launch_tc_leaf(const TcLeafArgs& a, int nrhs, cudaStream_t st);

// One launch per kind and rows bucket; asynchronous on st.
cudaError_t launch_tc(TcKind kind, const TcLaunch& a, cudaStream_t st);
// in[p * 64 + r] = split(x[perm[p] + r * ld_x]) (x in caller order, column major FP32), p < n,
// r < nrhs (<= 64); columns r >= nrhs are zero
cudaError_t launch_tc_gather(const float* x, int64_t ld_x, int nrhs, const int64_t* perm, int64_t n, uint32_t* in,
                             cudaStream_t st);
// y_out[perm[p] + r * ld_out] = sum over slots s of y[(s * n + p) * 64 + r], r < nrhs
cudaError_t launch_tc_combine(const float* y, int nslots, int64_t n, const int64_t* perm, float* out,
                              int64_t ld_out, int nrhs, cudaStream_t st);
// z of split z groups: in[zpos * 64 + r] = zscale * sum over the group's part blocks
cudaError_t launch_tc_zfix(const TcZFix* fix, int nfix, int max_rows, const TcZRow* rows, const float* zpart,
                           uint32_t* in, cudaStream_t st);
// adds split panels' partial row blocks (kTcRows rows each) into their output rows
cudaError_t launch_tc_fix(const Panel* panels, const PanelFix* fix, int nfix, const float* part, float* y,
                          cudaStream_t st);

}  // namespace hodlr
