// sums.cuh -- sums of the rows that chunk boundaries cut, in a fixed order.
//
// A walk over chunks of consecutive units leaves, per chunk and level, a head
// row (the partial sum of a node or output row that began before the chunk
// and ends in it) and a tail row (of the one that goes on in the next chunk).
// A chain is the run of chunk boundaries that cut one node: boundaries first
// .. last (boundary c lies before chunk c) give the partials tail(first - 1),
// .., tail(last - 1), head(last), which are added in this order in FP64.
#pragma once

#include "common.cuh"

namespace adatm {

struct SpanSums {
  uint32_t nchains = 0, ngroups = 0, nmids = 0;
  DevBuf<uint32_t> chain;        // kChainWords per chain
  DevBuf<uint32_t> group_chain;  // chain of every group
  DevBuf<double> gsum, msum;     // sums of the groups, and of the groups of groups (ldr each)
  DevBuf<uint32_t> arrived;      // children summed so far, per group of groups, then per chain
};

// Where the sums go: memo rows of each level, and the output rows of level 0
// (row out_ids[node], or row `node` without out_ids).
struct SpanTarget {
  float *store[kMaxModes] = {nullptr};
  double *out = nullptr;
  const uint32_t *out_ids = nullptr;
};

// The chains of nlev x nch boundaries: cut[k * nch + c] is 1 + the node that
// boundary c cuts at the k-th level (level_of[k]), or 0 where it cuts none
// (c = 0 never does). Device work; two counts come back to the host.
void span_prepare(SpanSums &s, const uint32_t *cut, int nlev, const int *level_of, uint32_t nch, int ldr,
                  cudaStream_t stream);

// Add the chains of span (per chunk, level slot, head and tail: ldr values).
template <typename T>
void span_launch(const SpanSums &s, const T *span, int nlev, int R, int ldr, const SpanTarget &t,
                 cudaStream_t stream);

inline int span_kernels(const SpanSums &s) { return s.nchains ? 1 : 0; }

}  // namespace adatm
