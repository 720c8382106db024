// mttkrp.cu -- tree-walk MTTKRP kernels (see mttkrp.cuh for the scheme).
#include <algorithm>
#include <type_traits>
#include <vector>

#include "mttkrp.cuh"
#include "rows.cuh"

namespace adatm {

namespace {

struct WalkArgs {
  int N, S, d, R, ldr;
  uint32_t chunk, nchunks;
  uint64_t nunits;
  uint64_t nfibs[kMaxModes];
  uint64_t dims[kMaxModes];    // rows of each level's factor
  const uint32_t *fptr[kMaxModes];
  const uint32_t *fids[kMaxModes];
  const float *vals;
  const float *src_rows;       // memo rows of the source level (S < N-1)
  const uint32_t *src_ids;     // fids of the source level
  const uint8_t *src_cd;       // close depths of the source level (S >= 1)
  const void *U[kMaxModes];
  float *store[kMaxModes];
  double *out;                 // MTTKRP output rows (FP64 sums)
  const uint32_t *sched;
  uint32_t *counter;           // chunks claimed so far (zeroed before each launch)
  const uint8_t *hot_slot;     // scatter: slot of an output row summed per block, 0xFF = none
  const uint32_t *hot_rows;    // scatter: output row of each slot
  int nhot;
  // contraction: the partial sums of the nodes a chunk boundary cuts go to per-chunk rows (head: the node that
  // began before the chunk and closes in it; tail: the node open at its
  // end), summed later in chunk order; span_lev[l] is level l's slot
  // (-1 = none)
  float *span;
  int span_nlev;
  int span_lev[kMaxModes];
};

// Row of chunk c's head (which = 0) or tail (which = 1) partial at level l.
__device__ __forceinline__ float *span_row(const WalkArgs &a, uint32_t c, int l, int which) {
  return a.span + (((size_t)c * a.span_nlev + a.span_lev[l]) * 2 + which) * a.ldr;
}

constexpr int kHotRows = 32;     // output rows summed per block, at most
constexpr uint32_t kHotMin = 32768;  // units that must hit a row to make it one
constexpr uint32_t kScatterChunk = 128;  // rows per warp of a contraction's scatter
constexpr uint64_t kHotScanRows = 1ull << 24;  // output rows the hot-row search examines, at most

constexpr int kWarps = 8;   // warps per block
constexpr int kBatch = 32;  // units per batch of a scatter or pull warp

// ---------------------------------------------------------------------------
// Contraction (S > d).
//
// A warp runs W independent walkers of L = 32 / W lanes with VW columns per
// lane; each walker walks its own chunk of consecutive source units, so one
// warp instruction advances W units and nothing is exchanged between walkers.
// Where a node closes is read from the tree's close depths (no fptr traffic):
// a unit with close depth c closes its ancestors at levels S-1 .. S-c.
//
// FOLD F (levels S-1 .. S-F are not stored and lie below d; at most
// kMaxFold): the nodes of those levels are not formed. Each unit's row is
// multiplied by the factor rows of its ancestors at levels S-1 .. S-F and
// summed straight into the open node of level top = S-1-F (acc). The
// ancestors of a batch's units are consecutive nodes from each level's open
// node on (a unit's is the open node plus the closes of that level before
// it), so their ids come with one coalesced load per level.
//
// Rounding: where several walkers share a warp, a batch's units are added to
// one another first and the batch's sum then to the open node's (`held`). One
// run over a chunk of c units is off by about u c / sqrt(3 N) of a row of N
// units, runs of B by u sqrt((B^2 + c^2 / B) / 3 N). A unit's value is multiplied
// into its first row before the others are: in a skewed tensor many units share
// rows, and what a product of rows alone is off by would not average out. (Up
// to three BF16 rows come first: their product is exact in FP32.) Errors of the
// root walks against FP64, with one run and the value last / as here: the
// 6th-order Zipf(1.3) tensor 3.4e-9, 4.6e-9, 8.7e-9 / 1.3e-9, 1.1e-9, 7.8e-10; the
// 5th-order one, BF16 rows, 5.6e-9, 4.7e-9 / 1.8e-9, 2.2e-9. It costs these walks
// 2.18, 2.04, 1.86 -> 2.22, 2.08, 1.90 ms and 2.26, 1.15 -> 2.30, 1.16 ms; with the
// sum held in registers, 2.26, 2.11, 1.91 and 2.41, 1.19.
//
// A node of level top that closes leaves the unit loop: its sum is stored
// (memo rows, outputs), or multiplied by its own factor row and added to the
// open node of the level above, in shared memory, and so on up as far as the
// unit closes. The sums of the nodes that a chunk boundary cuts go to
// per-chunk head and tail rows (sums.cuh adds them).
//
// What bounds it: the L1 data pipe and the latency of the gathers behind it,
// not DRAM. A row of R = 32 columns takes one of its cycles, so a unit takes
// F + 1, next to about two for the staging and the closes. On the 6th-order
// Zipf(1.3) tensor at 10.4M nonzeros (R = 32, F = 3) the pipe is busy 68% of
// the time at 19 warp instructions per nonzero (issue 50%): 0.38 ms, against
// 0.47 ms and 29 instructions for one walk per warp whose closes went through
// shared-memory items; the 77.9M-nonzero tensor's three contractions 2.22 /
// 2.08 / 1.90 ms against 2.62 / 2.43 / 2.23. Measured and not kept, when the first
// of these took 2.31 ms: rows of the folded levels kept across units and loaded
// under a predicate (a load with inactive lanes costs the pipe as much as a
// full one), one unit in flight with the next one's rows loaded ahead (2.33),
// three or five blocks per SM (2.46 / 2.48), two walkers of two columns per lane
// (3.26).
// ---------------------------------------------------------------------------
constexpr int kMaxFold = 5;
constexpr uint32_t kNoneHeld = 1u << 31;

template <int W>
struct WalkShape {
  static constexpr int L = 32 / W;            // lanes per walker
  static constexpr int B = L < 16 ? 16 : 32;   // units per walker and batch
  static constexpr int RD = B / L;            // staging rounds per batch
};

// Shared memory of one warp: the batch's staged units (a uint4 per unit: its
// row, its parent's row, its value twice, as the packed products take it;
// the rows of the ancestors further up in X words), one spare slot per walker,
// so that walkers read different banks; the units' close depths (a byte each,
// in the spare slot where they fit); the open nodes (a word per lane) and open
// sums (VW columns per lane) of levels d .. top-1; level top's sum of the
// batches before (several walkers).
__host__ __device__ constexpr int stage_words(int F) { return F <= 1 ? 0 : (F == 2 ? 1 : (F == 3 ? 2 : 4)); }
template <int W>
__host__ __device__ constexpr size_t depth_bytes() {
  return WalkShape<W>::B > (int)sizeof(uint4) ? (size_t)W * WalkShape<W>::B : 0;
}
template <int W, int VW, int F>
__host__ __device__ constexpr size_t contract_warp_smem(int d, int top) {
  return (size_t)W * (WalkShape<W>::B + 1) * (sizeof(uint4) + stage_words(F) * sizeof(uint32_t)) / 16 * 16 + 16 +
         depth_bytes<W>() + (size_t)(top > d ? top - d : 0) * 32 * (sizeof(uint32_t) + VW * sizeof(float)) +
         (W > 1 ? 32 * VW * sizeof(float) : 0);
}

// What the unit loop reads: factor rows of the source and folded levels lie
// in one allocation, addressed by row number from its base.
struct HotArgs {
  const void *base;             // row 0
  uint32_t src_row;             // first row of the source level's factor
  uint32_t fold_row[kMaxFold];  // and of level S-1-f's
  const uint32_t *fold_ids[kMaxFold];
  const uint32_t *top_ids;
  const void *top_rows;         // factor of level top
  uint32_t top_last;            // its last node
  float *top_store;             // its memo rows
  int top_keep;                 // whether its sums are stored or output
};

template <int W, int VW, FactorType FT, bool LEAF, int F>
__global__ void __launch_bounds__(256, 4)
    k_contract(const __grid_constant__ WalkArgs a, const __grid_constant__ HotArgs hot) {
  static_assert(F >= 0 && F <= kMaxFold, "folded levels");
  constexpr int L = WalkShape<W>::L, B = WalkShape<W>::B, RD = WalkShape<W>::RD;
  constexpr uint32_t LM = L == 32 ? 0xFFFFFFFFu : (1u << L) - 1u;
  extern __shared__ __align__(16) unsigned char walk_raw[];
  const int S = a.S, d = a.d, top = a.S - 1 - F;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wk = lane / L, li = lane % L;
  unsigned char *wbase = walk_raw + (size_t)warp * contract_warp_smem<W, VW, F>(d, top);
  constexpr int X = stage_words(F);
  constexpr size_t kStageBytes =
      (size_t)W * (B + 1) * (sizeof(uint4) + X * sizeof(uint32_t)) / 16 * 16 + 16;
  uint4 *const stage = reinterpret_cast<uint4 *>(wbase) + wk * (B + 1);
  uint32_t *const stage2 =
      reinterpret_cast<uint32_t *>(reinterpret_cast<uint4 *>(wbase) + W * (B + 1)) + wk * (B + 1) * X;
  uint8_t *const scd =
      depth_bytes<W>() != 0 ? wbase + kStageBytes + wk * B : reinterpret_cast<uint8_t *>(stage + B);
  // sum of the open level-top node in the batches before this one
  Row<VW> *const held = reinterpret_cast<Row<VW> *>(wbase + kStageBytes + depth_bytes<W>()) + lane;
  // open node and open sum of level l in {d .. top-1}: nodes[l * 32], carry[l * 32]
  uint32_t *const nodes = reinterpret_cast<uint32_t *>(held - lane + (W > 1 ? 32 : 0)) + lane - d * 32;
  Row<VW> *const carry =
      reinterpret_cast<Row<VW> *>(nodes + (top > d ? top : d) * 32 - lane) + lane - d * 32;
  const int col = li * VW;
  const bool act = col < a.R;
  constexpr int esz = FT == FactorType::F32 ? 4 : 2;
  // row offsets are staged in units of four columns (32 bits number the rows of
  // any factor that fits the device)
  constexpr int kUnitShift = FT == FactorType::F32 ? 4 : 3;
  const uint32_t row_units = (uint32_t)a.ldr / 4u;
  // lanes past the rank read column 0 (their results are never stored)
  const uint32_t lane_off = (uint32_t)(act ? col : 0) * esz;
  const char *rows = static_cast<const char *>(hot.base) + lane_off;
  asm volatile("" : "+l"(rows));  // kept, not computed again at each load
  const uint32_t stride = (uint32_t)a.ldr * esz;

  // units whose rows are in flight together: as many as the registers hold
  constexpr int SB = VW <= 2 ? 4 : (F <= 3 ? 2 : 1);
  // folded rows multiplied into the source row before the value is
  constexpr int E = FT == FactorType::BF16 ? (F < 2 ? F : 2) : 0;
  // the first group of W chunks by the warp's place in the grid, the next
  // ones from a counter (a resident grid), claimed while the current one runs
  uint32_t group = blockIdx.x * kWarps + warp;
  const uint32_t ngroups = (a.nchunks + W - 1) / W;
  while (group < ngroups) {
    uint32_t claim = 0;
    if (a.counter != nullptr && lane == 0) claim = atomicAdd(a.counter, 1u);
    const uint32_t chunk_id = group * W + wk;
    const bool live = chunk_id < a.nchunks;
    const uint32_t *sc = a.sched + (size_t)(live ? chunk_id : 0u) * (S + 1);
    uint32_t part = sc[S] | kNoneHeld;  // levels whose open node began before the chunk
    uint32_t nt = sc[top];
    uint32_t nf[F >= 1 ? F : 1];  // open nodes of the folded levels
#pragma unroll
    for (int f = 0; f < F; ++f) nf[f] = sc[S - 1 - f];
    for (int l = d; l < top; ++l) {
      nodes[l * 32] = sc[l];
      carry[l * 32] = row_zero<VW>();
    }
    uint32_t idt = __ldg(hot.top_ids + nt);  // the open level-top node's id
    Row<VW> acc = row_zero<VW>();
    // The sum x of a closed node: to its memo row, or, if it began before the
    // chunk, to the chunk's head row; at the root output, to its output row.
    auto keep = [&](int l, float *store, uint32_t n, uint32_t id, const Row<VW> &x) {
      if ((part >> l) & 1u) {
        part &= ~(1u << l);
        if (act) *reinterpret_cast<Row<VW> *>(span_row(a, chunk_id, l, 0) + col) = x;
      } else {
        if (store != nullptr && act) *reinterpret_cast<Row<VW> *>(store + (size_t)n * (uint32_t)a.ldr + col) = x;
        if (l == 0 && a.out != nullptr) st_out<VW>(a.out, id, a.ldr, col, row_values(x), act);
      }
    };
    // A unit closes level top and `more` levels above it.
    auto close = [&](uint32_t more) {
      Row<VW> x = acc;
      if (W > 1 && !(part & kNoneHeld)) {
        x = row_add(*held, x);
        part |= kNoneHeld;
      }
      acc = row_zero<VW>();
      const uint32_t id = idt;
      if (hot.top_keep) keep(top, hot.top_store, nt, id, x);
      ++nt;
      if (top == d) {
        if (d == 0) idt = __ldg(hot.top_ids + min(nt, hot.top_last));
        return;
      }
      Row<VW> c = carry[(top - 1) * 32];
      const Row<VW> row = ld_row<VW, FT>(row_at(static_cast<const char *>(hot.top_rows) + lane_off, id, stride));
      idt = __ldg(hot.top_ids + min(nt, hot.top_last));
      row_fma(c, x, row);
      int l = top - 1;
      for (; more != 0u; --more) {
        carry[l * 32] = row_zero<VW>();
        const uint32_t n = nodes[l * 32];
        nodes[l * 32] = n + 1u;
        const uint32_t up = __ldg(a.fids[l] + n);
        if (a.span_lev[l] >= 0) keep(l, a.store[l], n, up, c);
        if (l == d) return;
        x = c;
        --l;
        c = carry[l * 32];
        row_fma(c, x, ld_row<VW, FT>(row_at(static_cast<const char *>(a.U[l + 1]) + lane_off, up, stride)));
      }
      carry[l * 32] = c;
    };
    const uint32_t u0 = live ? chunk_id * a.chunk : 0u;  // (units are numbered in 32 bits)
    const uint32_t left0 = live ? min(a.chunk, (uint32_t)a.nunits - u0) : 0u;
    for (uint32_t b0 = 0; b0 < a.chunk; b0 += B) {
      const int cnt = left0 > b0 ? (int)min((uint32_t)B, left0 - b0) : 0;
      if (!__any_sync(~0u, cnt > 0)) break;
      const uint32_t base = u0 + b0;
      // stage the batch; mt: the units that close level top
      uint32_t mt = 0u;
      {
        uint32_t id[RD], cd[RD], anc[RD][5];
        float v[RD];
#pragma unroll
        for (int r = 0; r < RD; ++r) {
          const int j = r * L + li;
          const bool in = j < cnt;
          id[r] = in ? ld_stream(a.src_ids + (base + j)) : 0u;
          v[r] = 0.f;
          if constexpr (LEAF) v[r] = in ? ld_stream(a.vals + (base + j)) : 0.f;
          cd[r] = in ? ld_stream(a.src_cd + (base + j)) : 0u;
        }
#pragma unroll
        for (int r = 0; r < RD; ++r) {
          const bool in = r * L + li < cnt;
          const uint32_t lt = (1u << li) - 1u;
#pragma unroll
          for (int f = 0; f < 5; ++f) {
            anc[r][f] = 0u;
            if (f < F) {
              const uint32_t m = (__ballot_sync(~0u, cd[r] >= (uint32_t)(f + 1)) >> (wk * L)) & LM;
              uint32_t &n = nf[f < F ? f : 0];
              if (in) anc[r][f] = (ld_stream(hot.fold_ids[f] + (n + __popc(m & lt))) + hot.fold_row[f]) * row_units;
              n += __popc(m);
            }
          }
          mt |= ((__ballot_sync(~0u, cd[r] >= (uint32_t)(F + 1)) >> (wk * L)) & LM) << (r * L);
        }
#pragma unroll
        for (int r = 0; r < RD; ++r) {
          const int j = r * L + li;
          const uint32_t vb = __float_as_uint(v[r]);
          stage[j] = make_uint4((id[r] + hot.src_row) * row_units, anc[r][0], vb, vb);
          if constexpr (X >= 1) stage2[j * X] = anc[r][1];
          if constexpr (X >= 2) stage2[j * X + 1] = anc[r][2];
          if constexpr (X >= 4) {
            stage2[j * X + 2] = anc[r][3];
            stage2[j * X + 3] = anc[r][4];
          }
          scd[j] = (uint8_t)cd[r];
        }
      }
      __syncwarp();
      // the unit loop, the same for every lane; only a close is a walker's own
      const uint32_t any = __reduce_or_sync(~0u, mt);
      const char *mrow = nullptr;
      if constexpr (!LEAF)
        mrow = reinterpret_cast<const char *>(a.src_rows + (uint64_t)base * (uint32_t)a.ldr + (act ? col : 0));
      auto run = [&](auto full) {
        constexpr bool FULL = decltype(full)::value;
#pragma unroll 1
        for (int k = 0; k < B; k += SB) {
          if (!FULL && !__any_sync(~0u, k < cnt)) break;
          RawRow<VW, FT> g[SB], t[SB][F >= 1 ? F : 1];
          RawRow<VW, FactorType::F32> m[LEAF ? 1 : SB];
          uint64_t v[LEAF ? SB : 1];
#pragma unroll
          for (int q = 0; q < SB; ++q) {
            // units past the walker's last are staged as row 0 and not added
            const uint4 e = stage[k + q];
            ld_row<VW, FT>(g[q], rows + ((uint64_t)e.x << kUnitShift));
            if constexpr (F >= 1) ld_row<VW, FT>(t[q][0], rows + ((uint64_t)e.y << kUnitShift));
            const uint32_t *e2 = stage2 + (k + q) * X;
            if constexpr (F >= 2) ld_row<VW, FT>(t[q][1], rows + ((uint64_t)e2[0] << kUnitShift));
            if constexpr (F >= 3) ld_row<VW, FT>(t[q][2], rows + ((uint64_t)e2[1] << kUnitShift));
            if constexpr (F >= 4) ld_row<VW, FT>(t[q][3], rows + ((uint64_t)e2[2] << kUnitShift));
            if constexpr (F >= 5) ld_row<VW, FT>(t[q][4], rows + ((uint64_t)e2[3] << kUnitShift));
            if constexpr (LEAF) {
              v[q] = pack2(__uint_as_float(e.z), __uint_as_float(e.w));
            } else {
              raw_zero<VW, FactorType::F32>(m[q]);
              if (FULL || k + q < cnt) ld_row<VW, FactorType::F32>(m[q], mrow);
              mrow += (uint32_t)a.ldr * 4u;
            }
          }
#pragma unroll
          for (int q = 0; q < SB; ++q) {
            Row<VW> y;
            if constexpr (!LEAF) {
              y = raw_row<VW, FactorType::F32>(m[q]);
            } else if constexpr (VW == 1) {
              float lo, hi;
              unpack2(v[q], lo, hi);
              y.w = lo;
            } else {
#pragma unroll
              for (int i = 0; i < VW / 2; ++i) y.w[i] = v[q];
            }
            Row<VW> x = raw_row<VW, FT>(g[q]);
#pragma unroll
            for (int f = 0; f < E; ++f) x = row_mul(x, raw_row<VW, FT>(t[q][f]));
            if constexpr (F > E) {
              y = row_mul(y, x);
#pragma unroll
              for (int f = E; f + 1 < F; ++f) y = row_mul(y, raw_row<VW, FT>(t[q][f]));
              x = raw_row<VW, FT>(t[q][F - 1]);
            }
            if (FULL || k + q < cnt) row_fma(acc, y, x);
            if ((any >> (k + q)) & 1u) {
              if ((mt >> (k + q)) & 1u) close((uint32_t)scd[k + q] - (uint32_t)(F + 1));
              __syncwarp();
            }
          }
        }
      };
      if (__all_sync(~0u, cnt == B)) run(std::true_type{});
      else run(std::false_type{});
      if (W > 1 && b0 + B < a.chunk) {
        if (!(part & kNoneHeld)) acc = row_add(*held, acc);
        *held = acc;
        part &= ~kNoneHeld;
        acc = row_zero<VW>();
      }
      __syncwarp();
    }
    // chunk end: the nodes that the last unit did not close go on in the next
    // chunk; their partial sums go to the tail rows, or into their parents'
    if (live) {
      const uint32_t lastcd = __ldg(a.src_cd + (u0 + left0 - 1u));
      // what the level holds, with what the level below adds
      Row<VW> x = W > 1 && !(part & kNoneHeld) ? row_add(*held, acc) : acc;
      for (int l = top; l >= d; --l) {
        if (l < top) x = row_add(x, carry[l * 32]);
        if (l < S - (int)lastcd) {
          const uint32_t n = l == top ? nt : nodes[l * 32];
          if (a.span_lev[l] >= 0 && act) *reinterpret_cast<Row<VW> *>(span_row(a, chunk_id, l, 1) + col) = x;
          if (l > d)
            x = row_mul(x, ld_row<VW, FT>(row_at(static_cast<const char *>(a.U[l]),
                                                 __ldg(a.fids[l] + n), stride) + lane_off));
        }
      }
    }
    __syncwarp();
    group = a.counter != nullptr ? gridDim.x * kWarps + __shfl_sync(~0u, claim, 0) : ngroups;
  }
}

// ---------------------------------------------------------------------------
// Scatter (S == d): every unit adds src(u) * P_{d-1} to output row
// fids[d][u], with P_{d-1} = Q * U_{d-1}[parent] and Q the prefix of the
// levels above the parent (it changes only where a unit closes two or more
// levels). Units are independent, so a warp takes 32 / W of them per step:
// W lanes per unit, 4 columns (one float4) per lane, vector atomics.
// Skewed modes send many units of a batch to the same output row, and the
// vector atomics on that row serialise; so a batch whose units repeat an
// output row first stages every unit's row in shared memory and lets the
// first unit of each repeated row add the group's sum with one atomic.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float4 lds4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void sts4(float *p, float4 v) { *reinterpret_cast<float4 *>(p) = v; }

// Per-warp shared memory, sized by the row width: prefix rows (kMaxModes x
// ldr), the batch's (id, value) pairs, parent ids, output-row groups and
// leaders, then the staged unit rows (kBatch x ldr).
__host__ __device__ constexpr size_t scatter_warp_bytes(int ldr) {
  return ((size_t)kMaxModes * ldr * sizeof(float) + kBatch * (sizeof(uint2) + 3 * sizeof(uint32_t)) +
          (size_t)kBatch * ldr * sizeof(float) + 15) / 16 * 16;
}

// Prefix rows (per column, all ldr columns; rows ldr floats apart) of levels
// lo..hi-1.
template <FactorType FT>
__device__ __noinline__ void scatter_prefix(const WalkArgs &a, float *preq, uint32_t nodeL, int lo,
                                            int hi, int lane) {
  const int c = 4 * lane;
  const bool act = c < a.ldr;
  for (int l = lo; l < hi; ++l) {
    const uint32_t n = __shfl_sync(~0u, nodeL, l);
    const bool valid = (uint64_t)n < a.nfibs[l];
    const uint32_t f = valid ? __ldg(a.fids[l] + n) : 0u;
    float4 row = ld_factor4<FT>(a.U[l], f, a.ldr, c, act && valid);
    if (l > 0 && act) {
      const float4 p = *reinterpret_cast<const float4 *>(preq + (l - 1) * a.ldr + c);
      row = make_float4(row.x * p.x, row.y * p.y, row.z * p.z, row.w * p.w);
    }
    if (act) *reinterpret_cast<float4 *>(preq + l * a.ldr + c) = row;
  }
}

template <int W, FactorType FT, bool LEAF, bool HOT>
__global__ void __launch_bounds__(256, HOT ? 3 : 1) k_scatter(const __grid_constant__ WalkArgs a) {
  constexpr int UPS = 32 / W;  // units per step
  extern __shared__ __align__(16) unsigned char walk_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char *wbase = walk_raw + (size_t)warp * scatter_warp_bytes(a.ldr);
  float *preq = reinterpret_cast<float *>(wbase);  // kMaxModes x ldr columns
  uint2 *ustage = reinterpret_cast<uint2 *>(preq + kMaxModes * a.ldr);
  uint32_t *pstage = reinterpret_cast<uint32_t *>(ustage + kBatch);
  uint32_t *gstage = pstage + kBatch;  // lanes sharing each unit's output row
  uint32_t *lstage = gstage + kBatch;  // units that lead a repeated row
  float *xs = reinterpret_cast<float *>(lstage + kBatch);  // staged unit rows
  const int slot = lane / W;
  const int col = 4 * (lane % W);
  const bool act = col < a.R;
  const int d = a.S;
  // hot output rows: summed by the block in shared memory, added to the
  // output once at the end (their atomics would otherwise queue on a few L2
  // lines); the grid is then resident and warps stride over the chunks
  double *hacc = HOT ? reinterpret_cast<double *>(walk_raw + kWarps * scatter_warp_bytes(a.ldr)) : nullptr;
  if constexpr (HOT) {
    for (int i = threadIdx.x; i < a.nhot * a.ldr; i += blockDim.x) hacc[i] = 0.0;
    __syncthreads();
  }
  auto emit = [&](uint32_t row, const float4 &x) {
    if constexpr (HOT) {
      const uint32_t sl = __ldg(a.hot_slot + row);
      if (sl != 0xFFu) {
        double *h = hacc + sl * a.ldr + col;
        atomicAdd(h, (double)x.x);
        atomicAdd(h + 1, (double)x.y);
        atomicAdd(h + 2, (double)x.z);
        atomicAdd(h + 3, (double)x.w);
        return;
      }
    }
    double *o = a.out + (size_t)row * a.ldr + col;
    atomicAdd(o, (double)x.x);
    atomicAdd(o + 1, (double)x.y);
    atomicAdd(o + 2, (double)x.z);
    atomicAdd(o + 3, (double)x.w);
  };
  // without hot rows the grid covers every chunk: one chunk per warp
  for (uint32_t chunk_id = blockIdx.x * kWarps + warp; chunk_id < a.nchunks;
       chunk_id = HOT ? chunk_id + gridDim.x * kWarps : a.nchunks) {
    const uint32_t *sc = a.sched + (size_t)chunk_id * (d + 1);
    uint32_t nodeL = lane < d ? sc[lane] : 0u;
    if (d >= 2) scatter_prefix<FT>(a, preq, nodeL, 0, d - 1, lane);
    __syncwarp();
    const uint64_t u0 = (uint64_t)chunk_id * a.chunk;
    const uint64_t u1 = min(u0 + a.chunk, a.nunits);
    for (uint64_t base = u0; base < u1; base += kBatch) {
      const int cnt = (int)min((uint64_t)kBatch, u1 - base);
      const bool in = lane < cnt;
      const uint32_t id = in ? __ldg(a.src_ids + base + lane) : 0u;
      float v = 0.f;
      if constexpr (LEAF) v = in ? __ldg(a.vals + base + lane) : 0.f;
      const uint32_t cd = (in && d >= 1) ? (uint32_t)__ldg(a.src_cd + base + lane) : 0u;
      const uint32_t M = __ballot_sync(~0u, cd >= 1u);
      const uint32_t M2 = __ballot_sync(~0u, cd >= 2u);
      // factor-row ids of the parents (level d-1) of this batch's units
      const uint32_t nodeP = d >= 1 ? __shfl_sync(~0u, nodeL, d - 1) : 0u;
      uint32_t pf = 0;
      if (d >= 1 && (uint64_t)nodeP + lane < a.nfibs[d - 1]) pf = __ldg(a.fids[d - 1] + nodeP + lane);
      ustage[lane] = make_uint2(id, __float_as_uint(v));
      pstage[lane] = pf;
      // units of this batch that repeat an output row
      const uint32_t grp = __match_any_sync(~0u, in ? id : 0xFFFFFFFFu);
      const bool lead = in && (grp & lanemask_lt()) == 0;
      const bool stage = __ballot_sync(~0u, in && !lead) != 0u;
      gstage[lane] = grp;
      __syncwarp();
      int k = 0;
      while (k < cnt) {
        const uint32_t rest = M2 & (~0u << k);
        const int deep = rest ? __ffs(rest) - 1 : 32;
        const int ke = min(deep, cnt - 1);
        float4 Q = make_float4(1.f, 1.f, 1.f, 1.f);
        if (d >= 2 && act) Q = *reinterpret_cast<const float4 *>(preq + (d - 2) * a.ldr + col);
        // four steps' row loads are issued before any of their products
        constexpr int ST = 4;
        for (int k0 = k; k0 <= ke; k0 += ST * UPS) {
          float4 r[ST];
          float4 m[LEAF ? 1 : ST];
#pragma unroll
          for (int t = 0; t < ST; ++t) {
            const int unit = k0 + t * UPS + slot;
            const bool ok = unit <= ke && act;
            r[t] = make_float4(1.f, 1.f, 1.f, 1.f);
            if (d >= 1) r[t] = ld_factor4<FT>(a.U[d - 1], pstage[__popc(M & ((1u << (unit & 31)) - 1u))],
                                              a.ldr, col, ok);
            if constexpr (!LEAF) m[t] = ld_rows4(a.src_rows, base + (unit & 31), a.ldr, col, ok);
          }
#pragma unroll
          for (int t = 0; t < ST; ++t) {
            const int unit = k0 + t * UPS + slot;
            const bool ok = unit <= ke && act;
            const uint2 e = ustage[unit & 31];
            const float4 p = d >= 1 ? make_float4(Q.x * r[t].x, Q.y * r[t].y, Q.z * r[t].z, Q.w * r[t].w)
                                    : r[t];
            float4 x;
            if constexpr (LEAF) {
              const float sv = __uint_as_float(e.y);
              x = make_float4(sv * p.x, sv * p.y, sv * p.z, sv * p.w);
            } else {
              x = make_float4(m[t].x * p.x, m[t].y * p.y, m[t].z * p.z, m[t].w * p.w);
            }
            if (ok) {
              if (stage) sts4(xs + (unit & 31) * a.ldr + col, x);
              else emit(e.x, x);
            }
          }
        }
        if (deep == ke) {
          // unit ke closes levels d-1 .. d-c (c >= 2): the levels above its
          // parent move on and Q is recomputed
          const int c = (int)__shfl_sync(~0u, cd, ke);
          if (lane >= d - c && lane < d - 1) nodeL += 1;
          if ((uint64_t)__shfl_sync(~0u, nodeL, d - c) < a.nfibs[d - c])
            scatter_prefix<FT>(a, preq, nodeL, d - c, d - 1, lane);
          __syncwarp();
        }
        k = ke + 1;
      }
      if (stage) {
        // one atomic per distinct output row: the leading unit sums its group
        __syncwarp();
        const uint32_t L = __ballot_sync(~0u, lead);
        if (lead) lstage[__popc(L & lanemask_lt())] = (uint32_t)lane;
        __syncwarp();
        const int nl = __popc(L);
        for (int i0 = 0; i0 < nl; i0 += UPS) {
          const int i = i0 + slot;
          if (i < nl && act) {
            const uint32_t u = lstage[i];
            uint32_t members = gstage[u];
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
            while (members) {
              const int m = __ffs(members) - 1;
              members &= members - 1u;
              const float4 x = lds4(xs + m * a.ldr + col);
              sum = make_float4(sum.x + x.x, sum.y + x.y, sum.z + x.z, sum.w + x.w);
            }
            emit(ustage[u].x, sum);
          }
        }
      }
      if (d >= 1 && lane == d - 1) nodeL += (uint32_t)__popc(M);
      __syncwarp();
    }
  }
  if constexpr (HOT) {
    __syncthreads();
    for (int i = threadIdx.x; i < a.nhot * a.ldr; i += blockDim.x) {
      const double v = hacc[i];
      if (v != 0.0) atomicAdd(a.out + (size_t)a.hot_rows[i / a.ldr] * a.ldr + i % a.ldr, v);
    }
  }
}

// Units per output row of a scatter walk (the ids of its level).
__global__ void k_row_count(const uint32_t *ids, uint64_t n, uint32_t rows, uint32_t *count) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t r = ids[i];
    if (r < rows) atomicAdd(count + r, 1u);
  }
}

// Schedule: for chunk c, the node of every level 0..S-1 that contains the
// chunk's first unit, and which of those nodes started before it.
__global__ void k_schedule(WalkArgs a, uint32_t *sched) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.nchunks) return;
  const int S = a.S;
  const uint64_t u0 = (uint64_t)c * a.chunk;
  uint32_t child = (uint32_t)u0;
  uint32_t mask = 0;
  bool below_partial = false;
  for (int l = S - 1; l >= 0; --l) {
    // largest n with fptr[l][n] <= child
    const uint32_t *fp = a.fptr[l];
    uint64_t lo = 0, hi = a.nfibs[l] - 1;
    while (lo < hi) {
      const uint64_t mid = (lo + hi + 1) >> 1;
      if (fp[mid] <= child)
        lo = mid;
      else
        hi = mid - 1;
    }
    const uint32_t n = (uint32_t)lo;
    const bool p = (fp[n] < child) || below_partial;
    if (p) mask |= 1u << l;
    below_partial = p;
    sched[(size_t)c * (S + 1) + l] = n;
    child = n;
  }
  sched[(size_t)c * (S + 1) + S] = mask;
}

// ---------------------------------------------------------------------------
// Cut nodes.
// ---------------------------------------------------------------------------
// The nodes that chunk boundaries cut: cut[k * nchunks + c] = 1 + the node of
// the k-th spanned level that began before chunk c, else 0.
__global__ void k_cut_nodes(WalkArgs a, uint32_t *cut) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= a.nchunks) return;
  const uint32_t *sc = a.sched + (size_t)c * (a.S + 1);
  for (int l = 0; l < a.S; ++l)
    if (a.span_lev[l] >= 0)
      cut[(size_t)a.span_lev[l] * a.nchunks + c] = (sc[a.S] >> l) & 1u ? sc[l] + 1u : 0u;
}

// Memo rows of level l, or the scratch rows of a contraction's level-d sums.
float *store_of(const TreeWalk &w, int l) {
  return l == w.out && w.level_store() && w.scratch ? w.scratch->level_rows.get() : w.store[l];
}

WalkArgs make_args(const TreeWalk &w, const LevelFactors *f, double *out) {
  WalkArgs a;
  const DevCsf &c = *w.csf;
  a.N = w.nmodes;
  a.S = w.src;
  a.d = w.out;
  a.R = w.R;
  a.ldr = w.ldr;
  a.chunk = w.chunk;
  a.nchunks = w.nchunks;
  a.nunits = w.nunits;
  for (int l = 0; l < kMaxModes; ++l) {
    a.nfibs[l] = c.nfibs[l];
    a.dims[l] = l < c.nmodes ? c.dims[c.dim_perm[l]] : 0;
    a.fptr[l] = c.fptr[l].get();
    a.fids[l] = c.fids[l].get();
    a.U[l] = f ? f->U[l] : nullptr;
    a.store[l] = store_of(w, l);
  }
  a.vals = c.vals32.get();
  a.src_rows = w.src_rows;
  a.src_ids = c.fids[w.src].get();
  a.src_cd = w.src >= 1 ? c.cdepth[w.src].get() : nullptr;
  a.out = out;
  a.sched = w.sched.get();
  a.counter = w.sched.get() ? w.sched.get() + (size_t)w.nchunks * (w.src + 1) : nullptr;
  a.nhot = w.nhot;
  a.hot_slot = w.hot_slot.get();
  a.hot_rows = w.hot_rows.get();
  a.span = w.span_nlev > 0 && w.scratch ? w.scratch->span.get() : nullptr;
  a.span_nlev = w.span_nlev;
  for (int l = 0; l < kMaxModes; ++l) a.span_lev[l] = w.span_lev[l];
  return a;
}

// Blocks of `kernel` that fit on the device at once with `smem` bytes each.
template <typename K>
unsigned resident_blocks(K kernel, int threads, size_t smem) {
  int dev = 0, sms = 0, per_sm = 0;
  ADATM_CUDA(cudaGetDevice(&dev));
  ADATM_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  ADATM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
  return (unsigned)std::max(1, sms * std::max(1, per_sm));
}

// The lowest factor of the source level and the f levels above it.
const void *hot_base(const WalkArgs &a, int f) {
  const char *b = static_cast<const char *>(a.U[a.S]);
  for (int i = 0; i < f; ++i) b = std::min(b, static_cast<const char *>(a.U[a.S - 1 - i]));
  return b;
}

template <int W, int VW, FactorType FT, bool LEAF, int F>
void launch_contract_v(const WalkArgs &a, bool resident, cudaStream_t s) {
  const size_t smem = kWarps * contract_warp_smem<W, VW, F>(a.d, a.S - 1 - F);
  auto kern = k_contract<W, VW, FT, LEAF, F>;
  const unsigned groups = (a.nchunks + W - 1) / W;
  unsigned blocks = (groups + kWarps - 1) / kWarps;
  WalkArgs b = a;
  const int top = a.S - 1 - F;
  HotArgs h = {};
  h.base = hot_base(a, F);
  const size_t stride = (size_t)a.ldr * (FT == FactorType::F32 ? 4 : 2);
  auto first_row = [&](int l) {
    return (uint32_t)((static_cast<const char *>(a.U[l]) - static_cast<const char *>(h.base)) / stride);
  };
  h.src_row = first_row(a.S);
  for (int f = 0; f < F; ++f) {
    h.fold_row[f] = first_row(a.S - 1 - f);
    h.fold_ids[f] = a.fids[a.S - 1 - f];
  }
  h.top_ids = a.fids[top];
  h.top_rows = a.U[top];
  h.top_last = (uint32_t)a.nfibs[top] - 1u;
  h.top_store = a.store[top];
  h.top_keep = a.span_lev[top] >= 0;
  if (resident) blocks = std::min(blocks, resident_blocks(kern, 256, smem));
  if (blocks * kWarps < groups) ADATM_CUDA(cudaMemsetAsync(b.counter, 0, sizeof(uint32_t), s));
  else b.counter = nullptr;  // a group of chunks for every warp: nothing to claim
  kern<<<blocks, 256, smem, s>>>(b, h);
}

// Levels folded into the source loop, from level S-1 up: levels that are
// neither stored nor the output, as long as they hold at most fold_units()
// source units per node on average: at higher fan-out the extra row per unit
// costs more than the closes it saves. `want` >= 0 caps the count.
//
// Measured (ms per MTTKRP, fold up to 4 / 10 / 30 units per node; the line lies
// next to the best of them): FP32, R = 32, the 6th-order tensor's second and
// third contractions 2.18 / 2.26 / 2.26 and 1.97 / 1.97 / 2.16; BF16 rows (half
// the L1 bytes per row), R = 64, the 5th-order tensor's second contraction 1.44 /
// 1.25 / 1.25.
template <FactorType FT>
constexpr double fold_units() {
  return FT == FactorType::F32 ? 5.0 : 10.0;
}
int fold_levels(const WalkArgs &a, int want, double units, size_t stride) {
  const int cap = want < 0 ? kMaxFold : std::min(want, kMaxFold);
  int f = 0;
  while (f < cap && a.S - 1 - f > a.d && a.store[a.S - 1 - f] == nullptr &&
         (want >= 0 || f == 0 || (double)a.nunits <= units * (double)a.nfibs[a.S - 1 - f]))
    ++f;
  // the unit loop addresses the rows of its levels from the lowest factor on,
  // in 32-bit units of four columns (a single factor that fits the device does)
  const uint64_t unit = stride / (uint64_t)(a.ldr / 4);
  auto numbered = [&](int n) {
    const char *b = static_cast<const char *>(hot_base(a, n));
    for (int l = a.S; l >= a.S - n; --l) {
      const uint64_t off = (uint64_t)(static_cast<const char *>(a.U[l]) - b);
      if (off % stride != 0 || off / unit + a.dims[l] * (uint64_t)(a.ldr / 4) > 0xFFFFFFFFull) return false;
    }
    return true;
  };
  while (f > 0 && !numbered(f)) --f;
  return f;
}

// The (W, VW) shapes the contraction is built for: W walkers per warp with VW
// columns per lane (32 / W lanes cover the rank).
#define ADATM_CONTRACT_SHAPES(X) \
  X(1, 1) X(1, 2) X(1, 4) X(2, 1) X(2, 2) X(2, 4) X(4, 1) X(4, 2) X(4, 4) X(8, 1) X(8, 2) X(8, 4)
// Folded levels beyond the second are built for the default shapes above rank
// 8 (four columns per lane).
constexpr int max_fold(int vw) { return vw == 4 ? kMaxFold : 2; }

// Columns per walker lane for W walkers at rank R (0 if W walkers cannot
// cover R with at most 4 columns per lane).
int walker_cols(int R, int W) {
  for (int vw : {1, 2, 4})
    if ((32 / W) * vw >= R) return vw;
  return 0;
}

template <FactorType FT, bool LEAF>
void launch_contract(int walkers, int fold, const WalkArgs &a, bool resident, cudaStream_t s) {
  const int vw = walker_cols(a.R, walkers);
  const int f = std::min(
      fold_levels(a, fold, fold_units<FT>(), (size_t)a.ldr * (FT == FactorType::F32 ? 4 : 2)), max_fold(vw));
#define ADATM_CONTRACT_CASE(W, VW)                                                      \
  if (walkers == W && vw == VW) {                                                       \
    if constexpr (max_fold(VW) > 2) {                                                   \
      if (f == 5) launch_contract_v<W, VW, FT, LEAF, 5>(a, resident, s);                \
      else if (f == 4) launch_contract_v<W, VW, FT, LEAF, 4>(a, resident, s);           \
      else if (f == 3) launch_contract_v<W, VW, FT, LEAF, 3>(a, resident, s);           \
    }                                                                                   \
    if (f == 2) launch_contract_v<W, VW, FT, LEAF, 2>(a, resident, s);                  \
    else if (f == 1) launch_contract_v<W, VW, FT, LEAF, 1>(a, resident, s);             \
    else if (f == 0) launch_contract_v<W, VW, FT, LEAF, 0>(a, resident, s);             \
    ADATM_LAUNCH();                                                                     \
    return;                                                                             \
  }
  ADATM_CONTRACT_SHAPES(ADATM_CONTRACT_CASE)
#undef ADATM_CONTRACT_CASE
  throw BadInput("no contraction kernel for " + std::to_string(walkers) + " walkers at rank " +
                 std::to_string(a.R));
}

template <int W, FactorType FT, bool LEAF>
void launch_scatter_w(const WalkArgs &a, unsigned blocks, cudaStream_t s) {
  if (a.nhot > 0) {
    // each block sums the hot rows once: as few blocks as fit at once
    const size_t smem = kWarps * scatter_warp_bytes(a.ldr) + (size_t)a.nhot * a.ldr * sizeof(double);
    blocks = std::min(blocks, resident_blocks(k_scatter<W, FT, LEAF, true>, 256, smem));
    k_scatter<W, FT, LEAF, true><<<blocks, 256, smem, s>>>(a);
  } else {
    k_scatter<W, FT, LEAF, false><<<blocks, 256, kWarps * scatter_warp_bytes(a.ldr), s>>>(a);
  }
}

template <FactorType FT, bool LEAF>
void launch_scatter(int w, const WalkArgs &a, unsigned blocks, cudaStream_t s) {
  switch (w) {
    case 4: launch_scatter_w<4, FT, LEAF>(a, blocks, s); break;
    case 8: launch_scatter_w<8, FT, LEAF>(a, blocks, s); break;
    case 16: launch_scatter_w<16, FT, LEAF>(a, blocks, s); break;
    case 32: launch_scatter_w<32, FT, LEAF>(a, blocks, s); break;
    default: throw BadInput("unsupported lanes per unit");
  }
  ADATM_LAUNCH();
}

}  // namespace

// As many walkers as cover the rank at four columns (one 16-byte load) per lane.
int default_walkers(int R) { return R <= 16 ? 8 : (R <= 32 ? 4 : (R <= 64 ? 2 : 1)); }

bool walkers_supported(int R, int W) {
  return (W == 1 || W == 2 || W == 4) && R <= 128 && walker_cols(R, W) != 0;
}

namespace {

// Scatter: lanes per unit (4 columns per lane).
int lanes_for_rank(int R) {
  if (R <= 16) return 4;
  if (R <= 32) return 8;
  if (R <= 64) return 16;
  if (R <= 128) return 32;
  throw BadInput("rank above 128 is not supported by the GPU kernels");
}

}  // namespace

void set_walk_attributes() {
  static bool done = false;
  if (done) return;
#define ADATM_ATTR_C0(W, VW, FT, LEAF, F)                                       \
  ADATM_CUDA(cudaFuncSetAttribute(k_contract<W, VW, FT, LEAF, F>,               \
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,  \
                                  (int)(kWarps * contract_warp_smem<W, VW, F>(0, kMaxModes - 2 - F))));
#define ADATM_ATTR_C1(W, VW, FT, LEAF)       \
  ADATM_ATTR_C0(W, VW, FT, LEAF, 0)          \
  ADATM_ATTR_C0(W, VW, FT, LEAF, 1)          \
  ADATM_ATTR_C0(W, VW, FT, LEAF, 2)          \
  if constexpr (max_fold(VW) > 2) {          \
    ADATM_ATTR_C0(W, VW, FT, LEAF, 3)        \
    ADATM_ATTR_C0(W, VW, FT, LEAF, 4)        \
    ADATM_ATTR_C0(W, VW, FT, LEAF, 5)        \
  }
#define ADATM_ATTR_CS(W, VW)                       \
  ADATM_ATTR_C1(W, VW, FactorType::F32, true)      \
  ADATM_ATTR_C1(W, VW, FactorType::F32, false)     \
  ADATM_ATTR_C1(W, VW, FactorType::BF16, true)     \
  ADATM_ATTR_C1(W, VW, FactorType::BF16, false)
#define ADATM_ATTR_S(W, FT, LEAF)                                                 \
  ADATM_CUDA(cudaFuncSetAttribute(k_scatter<W, FT, LEAF, false>,                  \
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,    \
                                  (int)(kWarps * scatter_warp_bytes(128))));      \
  ADATM_CUDA(cudaFuncSetAttribute(k_scatter<W, FT, LEAF, true>,                   \
                                  cudaFuncAttributeMaxDynamicSharedMemorySize,    \
                                  (int)(kWarps * scatter_warp_bytes(128) +        \
                                        kHotRows * 128 * sizeof(double))));
#define ADATM_ATTR_ALL(M, X)                \
  M(X, FactorType::F32, true)               \
  M(X, FactorType::F32, false)              \
  M(X, FactorType::BF16, true)              \
  M(X, FactorType::BF16, false)
  ADATM_CONTRACT_SHAPES(ADATM_ATTR_CS)
  ADATM_ATTR_ALL(ADATM_ATTR_S, 4)
  ADATM_ATTR_ALL(ADATM_ATTR_S, 8)
  ADATM_ATTR_ALL(ADATM_ATTR_S, 16)
  ADATM_ATTR_ALL(ADATM_ATTR_S, 32)
#undef ADATM_ATTR_ALL
#undef ADATM_ATTR_S
#undef ADATM_ATTR_CS
#undef ADATM_ATTR_C1
#undef ADATM_ATTR_C0
  done = true;
}

// ---------------------------------------------------------------------------
// Preparation and launch.
// ---------------------------------------------------------------------------
namespace {

// Span slots and chains of a contraction: the levels whose cut nodes are summed
// over chunks (stored levels, and level 0 when it is the output), and for
// each node a chunk boundary cuts, the run of chunks it spans. Contractions
// below the root also store their level-d sums for the pull or the scatter.
void prepare_spans(TreeWalk &w, cudaStream_t s) {
  const DevCsf &c = *w.csf;
  const int S = w.src, d = w.out;
  if (d > 0) {
    // the level-d sums are stored (level_store), then pulled (or, with atomics,
    // scattered) into the output rows
    if (!w.deterministic) {
      w.scatter = std::make_unique<TreeWalk>();
      TreeWalk &t = *w.scatter;
      t.csf = w.csf;
      t.R = w.R;
      t.ldr = w.ldr;
      t.src = t.out = d;
      t.chunk = kScatterChunk;
      walk_prepare(t, s);
    }
  }
  w.span_nlev = 0;
  for (int l = 0; l < kMaxModes; ++l) w.span_lev[l] = -1;
  for (int l = 0; l < S; ++l)
    if (w.stores(l) || (l == 0 && d == 0)) w.span_lev[l] = w.span_nlev++;
  if (w.nchunks == 0 || w.span_nlev == 0) return;
  DevBuf<uint32_t> cut((size_t)w.span_nlev * w.nchunks, s);
  k_cut_nodes<<<(w.nchunks + 255) / 256, 256, 0, s>>>(make_args(w, nullptr, nullptr), cut.get());
  ADATM_LAUNCH();
  int level_of[kMaxModes];
  for (int l = 0; l < S; ++l)
    if (w.span_lev[l] >= 0) level_of[w.span_lev[l]] = l;
  span_prepare(w.sums, cut.get(), w.span_nlev, level_of, w.nchunks, w.ldr, s);
}

void launch_sums(const TreeWalk &w, double *out, cudaStream_t s) {
  SpanTarget t;
  for (int l = 0; l < kMaxModes; ++l) t.store[l] = store_of(w, l);
  t.out = w.out == 0 ? out : nullptr;
  t.out_ids = w.csf->fids[0].get();
  span_launch<float>(w.sums, w.scratch->span.get(), w.span_nlev, w.R, w.ldr, t, s);
}

}  // namespace

// The output rows of a scatter walk hit by the most units (at most
// kHotRows, each by at least kHotMin units), and the row -> slot table.
void find_hot_rows(TreeWalk &w, cudaStream_t s) {
  const DevCsf &c = *w.csf;
  const uint64_t rows64 = c.dims[c.dim_perm[w.out]];
  // a count per output row, on the device and the host: outputs with more
  // rows than kHotScanRows keep the plain scatter
  if (rows64 == 0 || rows64 > kHotScanRows) return;
  const uint32_t rows = (uint32_t)rows64;
  DevBuf<uint32_t> count(rows, s);
  ADATM_CUDA(cudaMemsetAsync(count.get(), 0, rows * sizeof(uint32_t), s));
  const unsigned blocks = (unsigned)std::min<uint64_t>((w.nunits + 255) / 256, 4096);
  k_row_count<<<blocks, 256, 0, s>>>(c.fids[w.out].get(), w.nunits, rows, count.get());
  ADATM_LAUNCH();
  std::vector<uint32_t> h(rows);
  ADATM_CUDA(cudaMemcpyAsync(h.data(), count.get(), rows * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  ADATM_CUDA(cudaStreamSynchronize(s));
  std::vector<uint32_t> order(rows);
  for (uint32_t r = 0; r < rows; ++r) order[r] = r;
  const uint32_t k = std::min<uint32_t>(kHotRows, rows);
  std::partial_sort(order.begin(), order.begin() + k, order.end(),
                    [&](uint32_t x, uint32_t y) { return h[x] > h[y] || (h[x] == h[y] && x < y); });
  std::vector<uint32_t> hot;
  for (uint32_t i = 0; i < k; ++i)
    if (h[order[i]] >= kHotMin) hot.push_back(order[i]);
  if (hot.empty()) return;
  std::vector<uint8_t> slot(rows, 0xFF);
  for (size_t i = 0; i < hot.size(); ++i) slot[hot[i]] = (uint8_t)i;
  w.hot_slot.alloc(rows, s);
  w.hot_rows.alloc(hot.size(), s);
  ADATM_CUDA(cudaMemcpyAsync(w.hot_slot.get(), slot.data(), rows, cudaMemcpyHostToDevice, s));
  ADATM_CUDA(cudaMemcpyAsync(w.hot_rows.get(), hot.data(), hot.size() * sizeof(uint32_t),
                             cudaMemcpyHostToDevice, s));
  ADATM_CUDA(cudaStreamSynchronize(s));
  w.nhot = (int)hot.size();
}

// Source units per chunk where the caller names none. A scatter's chunk is a
// warp's; a contraction's is a walker's, and every walker slot of a resident
// grid (4 blocks of 8 warps per SM) should have work: one chunk per slot while
// that is at most kOnce units (all slots then run once, side by side), else
// chunks small enough that the last ones leave few slots idle and no smaller
// than their own sums pay for (fewer walkers per warp, wider rows: larger).
// Above kOnce it is an eighth of a slot's share, at most 80 units, or 128 where
// rows are wider than 32 columns. Nonzeros that give every slot more than 64
// such chunks take larger ones, up to 256 units: the head and tail rows of a
// chunk (two rows for every spanned level) then take no more memory per
// nonzero than chunks of 256 do, where a tensor comes near the device's size.
//
// Measured (us per MTTKRP sequence, chunks of 16 / 32 / 64 / 96 / 128): 1M
// units, R = 16 (26 units per slot) 98 / 83 / 93 / 116 / 128; 3.5M units, R = 32
// (185 per slot) 672 / 666 / 760 / 812 / 926; 13M units, R = 32 (700 per slot)
// 935 / 809 / 790 / 812 / 839; 70M units, R = 32 7352 / 6552 / 6291 / 6273 / 6303;
// 3.4M units, R = 100 (740 per slot) 854 / 707 / 676 / 671 / 690; 40M units, R =
// 64 6198 / 4960 / 4612 / 4532 / 4487. Around kOnce, one root walk of R = 32,
// chunks of 16 / 32 / 64 / 128 / one per slot: 97 per slot 66 / 70 / 86 / 81 / 78; 120
// 76 / 79 / 87 / 84 / 84; 130 79 / 82 / 95 / 109 / -; 208 115 / 110 / 122 / 143 / -; R = 64,
// 122 per slot 71 / 67 / 68 / 65 / 65; 132 74 / 70 / 73 / 86 / -. The 78M-nonzero
// tensor (4112 per slot) with 80 / 112 / 256: 6405, 6425, 6670; at 256 units a slot
// has 16 chunks there, and 64 where the rule names 256.
uint32_t auto_chunk(const TreeWalk &w) {
  if (w.src == w.out) return w.src == w.nmodes - 1 ? 2 * kScatterChunk : kScatterChunk;
  constexpr uint64_t kOnce = 128, kMinChunk = 16;
  const uint64_t most = w.R <= 32 ? 80 : 128, large = w.src == w.nmodes - 1 ? 256 : most;
  const uint64_t slots = kSms * 32ull * default_walkers(w.R);
  const uint64_t per_slot = (w.nunits + slots - 1) / slots;
  const uint64_t c = per_slot <= kOnce
                         ? per_slot
                         : std::max(std::min(most, per_slot / 8), std::min(large, per_slot / 64));
  return (uint32_t)std::max(kMinChunk, (c + 15) / 16 * 16);
}

// A chunk size that the caller names is a warp's work: the walkers of a
// contraction warp divide it, down to 16 units each. Given whole to each
// walker, large chunks leave most slots of a small tensor's grid idle. us per
// MTTKRP sequence, whole / divided, chunks of 256 and 1024: 20K nonzeros, R = 16
// 166 / 57 and 492 / 101; 3.5M nonzeros, R = 32 1002 / 759 and 2881 / 998.
uint32_t walker_chunk(uint32_t chunk, int walkers) {
  const uint32_t W = (uint32_t)walkers;
  return std::max(std::min(chunk, 16u), chunk / W + (chunk % W != 0));
}

void walk_prepare(TreeWalk &w, cudaStream_t s) {
  set_walk_attributes();
  const DevCsf &c = *w.csf;
  w.nmodes = c.nmodes;
  w.nunits = c.nfibs[w.src];
  if (w.chunk == 0)
    w.chunk = auto_chunk(w);
  else if (w.src > w.out)
    w.chunk = walker_chunk(w.chunk, w.walkers > 0 ? w.walkers : default_walkers(w.R));
  w.chunk = std::min(w.chunk, 1u << 30);  // offsets in a chunk are 32-bit numbers
  w.nchunks = (uint32_t)((w.nunits + w.chunk - 1) / w.chunk);
  w.sched.alloc((size_t)std::max<uint32_t>(w.nchunks, 1) * (w.src + 1) + 1, s);  // + the chunk counter
  w.nhot = 0;
  w.hot_slot.reset();
  w.hot_rows.reset();
  if (w.nchunks == 0) return;
  WalkArgs a = make_args(w, nullptr, nullptr);
  k_schedule<<<(w.nchunks + 255) / 256, 256, 0, s>>>(a, w.sched.get());
  ADATM_LAUNCH();
  if (w.src > w.out) prepare_spans(w, s);
  if (w.deterministic && (w.src == w.out || w.out > 0)) {
    w.pull = std::make_unique<PullWalk>();
    pull_prepare(*w.pull, c, w.out, w.src == w.out && w.src == w.nmodes - 1, w.R, w.ldr, s);
  }
  if (!w.deterministic && w.src == w.out && w.nunits >= kHotMin) find_hot_rows(w, s);
}

bool WalkScratch::holds(const TreeWalk &w) const {
  return span.n >= w.span_words() && level_rows.n >= w.level_words() && pull_span.n >= w.pull_words();
}

void WalkScratch::reserve(const TreeWalk &w, cudaStream_t s) {
  auto grow = [&](auto &buf, size_t n) {
    if (buf.n >= n) return;
    std::decay_t<decltype(buf)> b(n, s);  // (the walks keep what they have if this throws)
    ADATM_CUDA(cudaMemsetAsync(b.get(), 0, b.bytes(), s));
    buf = std::move(b);
  };
  grow(span, w.span_words());
  grow(level_rows, w.level_words());
  grow(pull_span, w.pull_words());
}

namespace {

// src_rows: the walk's source rows where they are not its own (scatter of a
// contraction's sums).
void launch(const TreeWalk &w, const LevelFactors &f, FactorType ft, const float *src_rows, double *out,
            cudaStream_t s) {
  if (w.nchunks == 0) return;
  if (w.deterministic && w.src == w.out) {
    pull_launch(*w.pull, f.U, ft, src_rows, w.scratch->pull_span.get(), out, s);
    return;
  }
  WalkArgs a = make_args(w, &f, w.src > w.out && w.out > 0 ? nullptr : out);
  a.src_rows = src_rows;
  const bool leaf = w.src == w.nmodes - 1;
  if (w.src > w.out) {
    const int wk = w.walkers > 0 ? w.walkers : default_walkers(w.R);
    if (ft == FactorType::F32) {
      if (leaf) launch_contract<FactorType::F32, true>(wk, w.fold, a, w.resident, s);
      else launch_contract<FactorType::F32, false>(wk, w.fold, a, w.resident, s);
    } else {
      if (leaf) launch_contract<FactorType::BF16, true>(wk, w.fold, a, w.resident, s);
      else launch_contract<FactorType::BF16, false>(wk, w.fold, a, w.resident, s);
    }
    launch_sums(w, out, s);
    if (w.scatter) launch(*w.scatter, f, ft, w.scratch->level_rows.get(), out, s);
    else if (w.pull)
      pull_launch(*w.pull, f.U, ft, w.scratch->level_rows.get(), w.scratch->pull_span.get(), out, s);
  } else {
    const unsigned blocks = (unsigned)((w.nchunks + kWarps - 1) / kWarps);
    const int lanes = lanes_for_rank(w.R);
    if (ft == FactorType::F32) {
      if (leaf) launch_scatter<FactorType::F32, true>(lanes, a, blocks, s);
      else launch_scatter<FactorType::F32, false>(lanes, a, blocks, s);
    } else {
      if (leaf) launch_scatter<FactorType::BF16, true>(lanes, a, blocks, s);
      else launch_scatter<FactorType::BF16, false>(lanes, a, blocks, s);
    }
  }
}

}  // namespace

void walk_launch(const TreeWalk &w, const LevelFactors &f, FactorType ft, double *out, cudaStream_t s) {
  launch(w, f, ft, w.src_rows, out, s);
}

bool walk_fills_output(const TreeWalk &w) {
  if (w.nchunks == 0) return false;
  if (w.pull) return w.pull->every_row;
  if (w.src == w.out || w.out > 0) return false;
  const int vw = walker_cols(w.R, w.walkers > 0 ? w.walkers : default_walkers(w.R));
  return w.csf->nfibs[0] == w.csf->dims[w.csf->dim_perm[0]] && (w.R % 4 == 0 || vw == 4);
}

int walk_kernels(const TreeWalk &w) {
  if (w.nchunks == 0) return 0;
  int k = 0;
  if (w.src > w.out) {
    k += 1;                                            // the contraction
    k += span_kernels(w.sums);                         // the cut nodes' sums
  }
  if (w.pull) k += pull_kernels(*w.pull);
  if (!w.deterministic && w.src == w.out) k += 1;      // the scatter
  if (w.scatter) k += walk_kernels(*w.scatter);
  return k;
}

double walk_compulsory_bytes(const TreeWalk &w, FactorType ft, const uint64_t *dims_of_level,
                             uint64_t out_rows) {
  const DevCsf &c = *w.csf;
  const int N = c.nmodes;
  const double R = w.R;
  const double bf = ft == FactorType::F32 ? 4.0 : 2.0;
  double b = 0;
  // structure: every level from 0 to S is traversed
  for (int l = 0; l <= w.src; ++l) {
    b += 4.0 * (double)c.nfibs[l];                         // fids
    if (l < w.src) b += 4.0 * (double)(c.nfibs[l] + 1);    // fptr
  }
  if (w.src == N - 1) b += 4.0 * (double)c.nnz;            // leaf values
  else b += 4.0 * R * (double)c.nfibs[w.src];              // memo rows read
  for (int l = 0; l < N; ++l)
    if (l <= w.src && l != w.out) b += bf * R * (double)dims_of_level[l];  // factors
  for (int l = 0; l < kMaxModes; ++l)
    if (w.stores(l)) b += 4.0 * R * (double)c.nfibs[l];    // memo rows written
  b += 8.0 * R * (double)out_rows;                         // output (FP64 rows)
  return b;
}

}  // namespace adatm
