// mttkrp.cuh -- the MTTKRP kernels on CSF trees and their launch plans.
//
// Every MTTKRP of the reference (plain root / internal / leaf, memo root,
// memo reuse; mttkrp.c:241-1682) is one of two tree walks over a source
// level S and an output level d of one CSF tree:
//
//  * contract (S > d): every unit of level S (a nonzero when S = N-1, else a
//    stored memo row T_S) is multiplied by its factor row and summed into its
//    level S-1 parent; a completed node of level l > d multiplies its sum by
//    its own factor row and adds it to its parent; a completed node of level
//    d is written to the output row fids[d][node] (d = 0), or to a row of its
//    own that is then pulled or scattered like a memo row. Completed nodes of
//    the levels listed in `store` are also written to memo rows.
//  * scatter (S == d): every unit u adds src(u) * P_{d-1} to output row
//    fids[d][u], P_{d-1} the product of the factor rows on the root path of
//    its parent (leaf MTTKRP when d = N-1, memo reuse at its stored level).
//
// Work is split into chunks of `chunk` consecutive source units, one chunk
// per walker (a group of lanes), so the split follows nonzeros, not root
// slices (the reference's omp schedule(dynamic,16) over slices,
// mttkrp.c:392, cannot balance a slice holding 16% of the nonzeros). The
// partial sums of nodes cut by a chunk boundary are added in chunk order.
#pragma once

#include <memory>

#include "csf_build.cuh"
#include "pull.cuh"
#include "sums.cuh"

namespace adatm {

// Factor row matrices of one tree, in level order (U[l] belongs to mode
// dim_perm[l]); fp32 or bf16 with leading dimension ldr.
struct LevelFactors {
  const void *U[kMaxModes] = {nullptr};
};

// Rows that a walk writes and reads within one launch sequence: head and tail
// rows of a contraction's chunks, the level-d sums of one below the root, head
// and tail rows of a pull's segments. Walks that run one after another on one
// stream share them. The padding columns, which no walk has to write, are zero.
struct WalkScratch {
  DevBuf<float> span;        // nchunks x span_nlev x 2 x ldr
  DevBuf<float> level_rows;  // nodes of level d x ldr
  DevBuf<double> pull_span;  // nsegs x 2 x ldr
  bool holds(const struct TreeWalk &w) const;
  // Room for w's rows as well (what was there is not kept).
  void reserve(const struct TreeWalk &w, cudaStream_t s);
};

struct TreeWalk {
  int nmodes = 0;
  int src = 0;                 // source level S
  int out = 0;                 // output level d
  int R = 0, ldr = 0;
  uint32_t chunk = 0;          // source units per chunk (0 = by size, walk_prepare)
  uint32_t nchunks = 0;
  uint64_t nunits = 0;         // nodes of level S
  const DevCsf *csf = nullptr;
  const float *src_rows = nullptr;           // memo rows of level S (S < N-1)
  float *store[kMaxModes] = {nullptr};       // memo rows written, per level
  DevBuf<uint32_t> sched;                    // nchunks x (S + 1), then the chunk counter
  bool resident = true;                      // contraction grid: resident blocks that claim
                                             // chunks (else a group of chunks per warp)
  int walkers = 0;                           // contraction: walkers per warp (1, 2 or 4; 0 =
                                             // default_walkers(R), up to 8)
  int fold = -1;                             // contraction: most unstored levels above the
                                             // source folded into its loop (0..2; -1 = as
                                             // many as the tree's fan-out suggests, up to 5)
  // Scatter walks: the output rows that the most units hit (at most
  // kHotRows, each hit by at least kHotMin units) are summed per block in
  // shared memory; hot_slot maps an output row to its slot (0xFF = none).
  int nhot = 0;
  DevBuf<uint8_t> hot_slot;
  DevBuf<uint32_t> hot_rows;
  // Nodes that chunk boundaries cut (contractions, every mode): their
  // partial sums go to per-chunk rows (span) and are summed per node in
  // chunk order and in FP64 (sums), so a node spanning thousands of chunks (a
  // skewed root slice) takes no long chain of FP32 atomics. Deterministic accumulation
  // pulls scatters, and the output of contractions below the root, per output
  // row in the order of a stable sort by output row: no float atomics
  // anywhere, so repeated runs agree bit for bit.
  bool deterministic = false;
  int span_nlev = 0;
  int span_lev[kMaxModes] = {-1, -1, -1, -1, -1, -1, -1, -1};
  SpanSums sums;
  std::unique_ptr<TreeWalk> scatter; // contraction below the root, with atomics: the
                                     // scatter of its level-d sums into the output rows
  std::unique_ptr<PullWalk> pull;    // scatter of level `out` as a pull (deterministic)
  std::shared_ptr<WalkScratch> scratch;  // set before the first launch
  // contraction below the root: its level-d sums are rows of the scratch
  bool level_store() const { return src > out && out > 0; }
  bool stores(int l) const { return store[l] != nullptr || (l == out && level_store()); }
  size_t span_words() const { return (size_t)nchunks * span_nlev * 2 * ldr; }
  size_t level_words() const { return level_store() ? (size_t)csf->nfibs[out] * ldr : 0; }
  size_t pull_words() const { return pull ? pull->span_words() : 0; }
};

// Kernel launches of one walk (for launch counts).
int walk_kernels(const TreeWalk &w);

// Walkers per warp of a contraction by default at rank R, and whether a
// caller may choose W walkers at rank R.
int default_walkers(int R);
bool walkers_supported(int R, int W);

// Fill the chunk schedule: node ids at levels 0..S-1 of every chunk's first
// unit, plus a bit mask of the levels whose node began before the chunk.
void walk_prepare(TreeWalk &w, cudaStream_t s);

// Whether the walk writes every value of its output rows, so that they need
// no clearing: every row has units, nothing is added with atomics, and the
// padding columns are written.
bool walk_fills_output(const TreeWalk &w);

// Launch the walk: output rows (FP64, dims x ldr) must be zero beforehand
// unless the walk fills them (the caller clears them).
void walk_launch(const TreeWalk &w, const LevelFactors &f, FactorType ft, double *out,
                 cudaStream_t s);

// Bytes the walk must move through HBM (structure read once, memo rows read
// or written once, factors read once, output written once): the compulsory
// traffic used for the roofline figure.
double walk_compulsory_bytes(const TreeWalk &w, FactorType ft, const uint64_t *dims_of_level,
                             uint64_t out_rows);

}  // namespace adatm
