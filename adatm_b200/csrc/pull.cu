// pull.cu -- MTTKRP pulls (see pull.cuh).
#include <algorithm>
#include <type_traits>

#include "pull.cuh"
#include "rows.cuh"

namespace adatm {

namespace {

constexpr int kWarps = 8;  // warps per block

struct PullArgs {
  int d, R, ldr;
  uint32_t n, seg, nsegs;
  const uint32_t *perm, *row;
  const float *vals;
  const uint32_t *anc[kMaxModes];  // nearest ancestor first (level d-1 down to 0)
  const void *U[kMaxModes];        // their factors
  const float *src_rows;
  double *out, *span;
};

// Shared memory of one warp: a uint4 per staged unit (its source row or
// value, the rows of its three nearest ancestors), and a second one where it
// has more; one spare slot per walker, so that walkers read different banks.
template <int W, int D>
struct PullShape {
  static constexpr int L = 32 / W;            // lanes per walker, four columns each
  static constexpr int B = L < 16 ? 16 : 32;  // units per walker and batch
  static constexpr int RD = B / L;            // staging rounds per batch
  static constexpr int slots = W * (B + 1);
  static constexpr size_t smem = (size_t)kWarps * slots * sizeof(uint4) * (D > 3 ? 2 : 1);
};

// A warp runs W independent walkers of L lanes (four columns, one 16-byte load
// per row and lane); each walks one segment of consecutive units, adds
// src * U_{d-1}[..] * .. * U_0[..] of each to FP64 sums in registers and
// stores a row's sum where the row ends. A row that a segment boundary cuts
// leaves its parts in the segments' head and tail rows (sums.cuh adds them in
// order), so long rows need no splitting of their own and all segments are
// alike. D is the number of ancestor levels, 4 standing for four or more.
//
// The ancestors' factor rows are gathered straight from the factors (they stay
// in L1 and L2) instead of from prefix rows formed beforehand: level by level
// those were as many rows as the level above has nodes, written and then read
// in random order from HBM.
//
// What bounds it: the source rows, read once in random order (row sources),
// and the latency behind them. Measured, with one
// unit per warp, prefix rows and rows packed into segments on the host, and
// now (us per MTTKRP): 16.1M rows of R = 64, two ancestor levels, BF16
// factors, 2553 and 846 (5.2 TB/s of source rows and indices); 4.5M rows of R = 32
// 445 and 148; 2.3M rows of R = 32 314 and 64; 0.6M rows of R = 16 68 and 24.
template <int W, FactorType FT, bool LEAF, int D>
__global__ void __launch_bounds__(256, 4) k_pull(const __grid_constant__ PullArgs a) {
  using S = PullShape<W, D>;
  constexpr int L = S::L, B = S::B, RD = S::RD;
  constexpr uint32_t LM = L == 32 ? 0xFFFFFFFFu : (1u << L) - 1u;
  constexpr int DD = D > 3 ? 3 : D;                      // ancestors in the first uint4
  constexpr int SB = D <= 1 ? 4 : (D <= 3 ? 2 : 1);      // units in flight
  extern __shared__ __align__(16) unsigned char pull_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wk = lane / L, li = lane % L, col = 4 * li;
  uint4 *const stage = reinterpret_cast<uint4 *>(pull_raw) + (size_t)warp * S::slots * (D > 3 ? 2 : 1) + wk * (B + 1);
  uint4 *const stage2 = stage + S::slots;  // D > 3 only
  const bool act = col < a.R;
  constexpr int esz = FT == FactorType::F32 ? 4 : 2;
  const uint32_t lane_off = (uint32_t)(act ? col : 0);
  const uint32_t stride = (uint32_t)a.ldr * esz, src_stride = (uint32_t)a.ldr * 4u;
  const char *const src = LEAF ? nullptr : reinterpret_cast<const char *>(a.src_rows + lane_off);
  const char *U[DD > 0 ? DD : 1];
#pragma unroll
  for (int f = 0; f < DD; ++f) U[f] = static_cast<const char *>(a.U[f]) + lane_off * esz;

  const uint32_t sg = (blockIdx.x * kWarps + warp) * W + wk;
  const bool live = sg < a.nsegs;
  const uint32_t jb = live ? sg * a.seg : 0u, je = live ? min(a.n - jb, a.seg) + jb : 0u;
  // the row of the first unit began in an earlier segment
  bool head = live && jb > 0u && __ldg(a.row + jb - 1u) == __ldg(a.row + jb);
  bool open = false;  // the last unit's row goes on in the next segment
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  auto put = [&](double *p) {
    if (act) {
      reinterpret_cast<double2 *>(p + col)[0] = make_double2(acc[0], acc[1]);
      reinterpret_cast<double2 *>(p + col)[1] = make_double2(acc[2], acc[3]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i] = 0.0;
  };
  for (uint32_t b0 = 0; b0 < a.seg; b0 += B) {
    const uint32_t base = jb + b0;
    const int cnt = live && base < je ? (int)min((uint32_t)B, je - base) : 0;
    if (!__any_sync(~0u, cnt > 0)) break;
    uint32_t ends = 0u;  // units that end their row
    {
      uint32_t x[RD], row[RD], next[RD], anc[RD][7];
#pragma unroll
      for (int r = 0; r < RD; ++r) {
        const uint32_t j = base + r * L + li;
        const bool in = r * L + li < cnt;
        if constexpr (LEAF) x[r] = in ? __float_as_uint(ld_stream(a.vals + j)) : 0u;
        else x[r] = in ? ld_stream(a.perm + j) : 0u;
        row[r] = in ? ld_stream(a.row + j) : 0u;
        next[r] = in && j + 1u < a.n ? __ldg(a.row + j + 1u) : ~0u;
#pragma unroll
        for (int f = 0; f < 7; ++f) {
          anc[r][f] = 0u;
          if (f < DD || (D > 3 && f < a.d)) anc[r][f] = in ? ld_stream(a.anc[f] + j) : 0u;
        }
      }
#pragma unroll
      for (int r = 0; r < RD; ++r) {
        const bool end = r * L + li < cnt && row[r] != next[r];
        ends |= ((__ballot_sync(~0u, end) >> (wk * L)) & LM) << (r * L);
        stage[r * L + li] = make_uint4(x[r], anc[r][0], anc[r][1], anc[r][2]);
        if constexpr (D > 3) stage2[r * L + li] = make_uint4(anc[r][3], anc[r][4], anc[r][5], anc[r][6]);
      }
    }
    __syncwarp();
    const uint32_t any = __reduce_or_sync(~0u, ends);
    auto run = [&](auto full) {
      constexpr bool FULL = decltype(full)::value;
#pragma unroll 1
      for (int k = 0; k < B; k += SB) {
        if (!FULL && !__any_sync(~0u, k < cnt)) break;
        RawRow<4, FactorType::F32> m[LEAF ? 1 : SB];
        RawRow<4, FT> t[SB][D > 0 ? (D > 3 ? 7 : DD) : 1];
        float v[LEAF ? SB : 1];
#pragma unroll
        for (int q = 0; q < SB; ++q) {
          // units past the segment's last read row 0 and are not added
          const uint4 e = stage[k + q];
          if constexpr (LEAF) v[q] = __uint_as_float(e.x);
          else ld_row_once(m[q], row_at(src, e.x, src_stride));
          if constexpr (DD >= 1) ld_row<4, FT>(t[q][0], row_at(U[0], e.y, stride));
          if constexpr (DD >= 2) ld_row<4, FT>(t[q][1], row_at(U[1], e.z, stride));
          if constexpr (DD >= 3) ld_row<4, FT>(t[q][2], row_at(U[2], e.w, stride));
          if constexpr (D > 3) {
            const uint4 e2 = stage2[k + q];
            const uint32_t id[4] = {e2.x, e2.y, e2.z, e2.w};
#pragma unroll
            for (int f = 3; f < 7; ++f)
              if (f < a.d)
                ld_row<4, FT>(t[q][f], row_at(static_cast<const char *>(a.U[f]) + lane_off * esz, id[f - 3], stride));
          }
        }
#pragma unroll
        for (int q = 0; q < SB; ++q) {
          Row<4> x;
          if constexpr (LEAF) x.w[0] = x.w[1] = pack2(v[q], v[q]);
          else x = raw_row<4, FactorType::F32>(m[q]);
          // the value or source row times the nearest ancestor's row first: units
          // that share ancestors then do not share the rounding of a product of
          // theirs; up to three BF16 rows come first, their product is exact
          if constexpr (FT == FactorType::BF16 && DD >= 2) {
            Row<4> e = raw_row<4, FT>(t[q][0]);
#pragma unroll
            for (int f = 1; f < DD; ++f) e = row_mul(e, raw_row<4, FT>(t[q][f]));
            x = row_mul(x, e);
          } else {
#pragma unroll
            for (int f = 0; f < DD; ++f) x = row_mul(x, raw_row<4, FT>(t[q][f]));
          }
          if constexpr (D > 3)
#pragma unroll
            for (int f = 3; f < 7; ++f)
              if (f < a.d) x = row_mul(x, raw_row<4, FT>(t[q][f]));
          if (FULL || k + q < cnt) {
            const fv<4> y = row_values(x);
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[i] += (double)y.x[i];
          }
          if ((any >> (k + q)) & 1u) {
            if ((ends >> (k + q)) & 1u) {
              put(head ? a.span + (size_t)sg * 2 * a.ldr : a.out + (size_t)__ldg(a.row + base + k + q) * a.ldr);
              head = false;
            }
            __syncwarp();
          }
        }
      }
    };
    if (__all_sync(~0u, cnt == B)) run(std::true_type{});
    else run(std::false_type{});
    if (cnt > 0) open = !((ends >> (cnt - 1)) & 1u);
    __syncwarp();
  }
  if (open) put(a.span + ((size_t)sg * 2 + 1) * a.ldr);
}

// flags[i] = whether unit i ends its parent (its exclusive prefix sum is the
// unit's parent).
__global__ void k_last_child(const uint8_t *cd, uint64_t n, uint32_t *flags) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) flags[i] = cd[i] >= 1u;
}

struct AncArgs {
  int d;
  const uint32_t *parent[kMaxModes];  // parent of every node of levels 1 .. d
  const uint32_t *fids[kMaxModes];
  uint32_t *anc[kMaxModes];           // by level
};

__global__ void k_ancestors(const uint32_t *perm, uint64_t n, AncArgs a, const float *vals_in, float *vals) {
  const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  uint32_t p = perm[j];
  if (vals) vals[j] = vals_in[p];
  for (int l = a.d; l >= 1; --l) {
    p = a.parent[l][p];
    a.anc[l - 1][j] = a.fids[l - 1][p];
  }
}

// Units that begin an output row (their number is the number of rows hit).
__global__ void k_count_rows(const uint32_t *row, uint64_t n, uint32_t *count) {
  const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t b = __ballot_sync(~0u, j < n && (j == 0 || row[j] != row[j - 1]));
  if ((threadIdx.x & 31) == 0 && b != 0u) atomicAdd(count, (uint32_t)__popc(b));
}

// cut[s] = 1 + the row that the boundary before segment s cuts, or 0.
__global__ void k_cut_rows(const uint32_t *row, uint32_t seg, uint32_t nsegs, uint32_t *cut) {
  const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsegs) return;
  const uint64_t j = (uint64_t)s * seg;
  cut[s] = s > 0u && row[j - 1] == row[j] ? row[j] + 1u : 0u;
}

unsigned blocks_of(uint64_t n) { return (unsigned)((n + 255) / 256); }

int walkers_of(int R) { return R <= 16 ? 8 : (R <= 32 ? 4 : (R <= 64 ? 2 : 1)); }

template <int W, FactorType FT, bool LEAF>
void launch(const PullArgs &a, cudaStream_t s) {
  const unsigned blocks = (unsigned)(((uint64_t)a.nsegs + kWarps * W - 1) / (kWarps * W));
  switch (std::min(a.d, 4)) {
    case 0: k_pull<W, FT, LEAF, 0><<<blocks, 256, PullShape<W, 0>::smem, s>>>(a); break;
    case 1: k_pull<W, FT, LEAF, 1><<<blocks, 256, PullShape<W, 1>::smem, s>>>(a); break;
    case 2: k_pull<W, FT, LEAF, 2><<<blocks, 256, PullShape<W, 2>::smem, s>>>(a); break;
    case 3: k_pull<W, FT, LEAF, 3><<<blocks, 256, PullShape<W, 3>::smem, s>>>(a); break;
    default: k_pull<W, FT, LEAF, 4><<<blocks, 256, PullShape<W, 4>::smem, s>>>(a); break;
  }
  ADATM_LAUNCH();
}

template <FactorType FT, bool LEAF>
void launch_w(const PullArgs &a, cudaStream_t s) {
  switch (walkers_of(a.R)) {
    case 8: launch<8, FT, LEAF>(a, s); break;
    case 4: launch<4, FT, LEAF>(a, s); break;
    case 2: launch<2, FT, LEAF>(a, s); break;
    default: launch<1, FT, LEAF>(a, s); break;
  }
}

}  // namespace

void pull_prepare(PullWalk &p, const DevCsf &c, int d, bool leaf, int R, int ldr, cudaStream_t s) {
  if (R > 128) throw BadInput("rank above 128 is not supported by the GPU kernels");
  p.d = d;
  p.R = R;
  p.ldr = ldr;
  p.leaf = leaf;
  p.n = c.nfibs[d];
  p.nsegs = 0;
  p.every_row = false;
  if (p.n == 0) return;
  sort_by_row(c.fids[d].get(), p.n, c.dims[c.dim_perm[d]], p.perm, p.row, s);
  AncArgs a = {};
  a.d = d;
  DevBuf<uint32_t> parent[kMaxModes];
  for (int l = 1; l <= d; ++l) {
    const uint64_t n = c.nfibs[l];
    DevBuf<uint32_t> flags(n, s), tmp(scan_tmp_words(n), s);
    parent[l].alloc(n, s);
    k_last_child<<<blocks_of(n), 256, 0, s>>>(c.cdepth[l].get(), n, flags.get());
    ADATM_LAUNCH();
    exclusive_scan_u32(flags.get(), parent[l].get(), n, tmp.get(), s);
    a.parent[l] = parent[l].get();
  }
  for (int l = 0; l < d; ++l) {
    p.anc[l].alloc(p.n, s);
    a.anc[l] = p.anc[l].get();
    a.fids[l] = c.fids[l].get();
  }
  if (leaf) p.vals.alloc(p.n, s);
  k_ancestors<<<blocks_of(p.n), 256, 0, s>>>(p.perm.get(), p.n, a, c.vals32.get(), leaf ? p.vals.get() : nullptr);
  ADATM_LAUNCH();
  // segments: one per walker slot of a full device while that is at most 128
  // units, else short enough that the last ones leave few slots idle. Leaf
  // pulls, us with 16 / 32 / 64 / 128 / one per slot: R = 32, 97 units per slot 61 /
  // 62 / 61 / 65 / 61; 120 75 / 72 / 67 / 68 / 68; 130 78 / 76 / 75 / 84 / -; 208 115 / 112 /
  // 113 / 105 / -; 460 238 / 212 / 209 / 209 / -; R = 64, 132 per slot 76 / 70 / 73 / 84 / -
  const uint64_t slots = kSms * 32ull * walkers_of(R), per_slot = (p.n + slots - 1) / slots;
  const uint64_t u = per_slot <= 128 ? per_slot : std::min<uint64_t>(128, per_slot / 4);
  p.seg = (uint32_t)std::max<uint64_t>(16, (u + 15) / 16 * 16);
  p.nsegs = (uint32_t)((p.n + p.seg - 1) / p.seg);
  DevBuf<uint32_t> cut(p.nsegs, s), hit(1, s);
  ADATM_CUDA(cudaMemsetAsync(hit.get(), 0, sizeof(uint32_t), s));
  k_count_rows<<<blocks_of(p.n), 256, 0, s>>>(p.row.get(), p.n, hit.get());
  ADATM_LAUNCH();
  uint32_t rows_hit = 0;
  ADATM_CUDA(cudaMemcpyAsync(&rows_hit, hit.get(), sizeof(rows_hit), cudaMemcpyDeviceToHost, s));
  k_cut_rows<<<blocks_of(p.nsegs), 256, 0, s>>>(p.row.get(), p.seg, p.nsegs, cut.get());
  ADATM_LAUNCH();
  const int level = 0;
  span_prepare(p.sums, cut.get(), 1, &level, p.nsegs, ldr, s);  // (waits for the count as well)
  p.every_row = rows_hit == c.dims[c.dim_perm[d]];
  if (leaf) p.perm.reset();
}

void pull_launch(const PullWalk &p, const void *const *U, FactorType ft, const float *src_rows, double *span,
                 double *out, cudaStream_t s) {
  if (p.nsegs == 0) return;
  PullArgs a = {};
  a.d = p.d;
  a.R = p.R;
  a.ldr = p.ldr;
  a.n = (uint32_t)p.n;
  a.seg = p.seg;
  a.nsegs = p.nsegs;
  a.perm = p.perm.get();
  a.row = p.row.get();
  a.vals = p.vals.get();
  for (int f = 0; f < p.d; ++f) {
    a.anc[f] = p.anc[p.d - 1 - f].get();
    a.U[f] = U[p.d - 1 - f];
  }
  a.src_rows = src_rows;
  a.out = out;
  a.span = span;
  if (ft == FactorType::F32) {
    if (p.leaf) launch_w<FactorType::F32, true>(a, s);
    else launch_w<FactorType::F32, false>(a, s);
  } else {
    if (p.leaf) launch_w<FactorType::BF16, true>(a, s);
    else launch_w<FactorType::BF16, false>(a, s);
  }
  SpanTarget t;
  t.out = out;
  span_launch<double>(p.sums, span, 1, p.R, p.ldr, t, s);
}

int pull_kernels(const PullWalk &p) { return p.nsegs ? 1 + span_kernels(p.sums) : 0; }

}  // namespace adatm
