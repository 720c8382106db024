// pull.cuh -- MTTKRP scatters as pulls: the units of a level in a stable order
// by output row, so every output row is summed in a fixed order, in FP64, and
// written once.
#pragma once

#include "csf_build.cuh"
#include "sums.cuh"

namespace adatm {

enum class FactorType : int { F32 = 0, BF16 = 1 };

struct PullWalk {
  int d = 0, R = 0, ldr = 0;
  bool leaf = false;             // units are nonzeros (else rows of level d)
  uint64_t n = 0;                // units
  uint32_t seg = 0, nsegs = 0;   // units per segment (a walker's)
  DevBuf<uint32_t> perm;         // unit (row sources)
  DevBuf<float> vals;            // value (leaf sources)
  DevBuf<uint32_t> row;          // output row
  DevBuf<uint32_t> anc[kMaxModes];  // factor row of the ancestor at levels 0 .. d-1
  SpanSums sums;                 // of the rows that segment boundaries cut
  bool every_row = false;        // every output row has units
  size_t span_words() const { return (size_t)nsegs * 2 * ldr; }
};

// Sort level d's units by output row and look their ancestors up (device work).
void pull_prepare(PullWalk &p, const DevCsf &c, int d, bool leaf, int R, int ldr, cudaStream_t s);

// out[row] = sum over the row's units of src(unit) times the factor rows of
// its ancestors (U: factor rows per level); rows without units are left alone.
// span: head and tail row of every segment (span_words(), padding columns zero).
void pull_launch(const PullWalk &p, const void *const *U, FactorType ft, const float *src_rows, double *span,
                 double *out, cudaStream_t s);

int pull_kernels(const PullWalk &p);

}  // namespace adatm
