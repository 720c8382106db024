// sums.cu -- ordered sums of cut rows (see sums.cuh).
#include <type_traits>

#include "sums.cuh"

namespace adatm {

namespace {

constexpr uint32_t kGroup = 64;  // partials that one walker (a group of lanes) adds
constexpr uint32_t kMid = 64;    // groups under one group of groups, and most groups of a chain without
constexpr uint32_t kWideGroups = kSms * 64;
// words of a chain: level, node, level slot, first boundary, partials, first
// group, first group of groups, groups of groups (0 where the groups are few)
constexpr int kChainWords = 8;

struct CutArgs {
  int nlev;
  int level_of[kMaxModes];
  uint32_t nch;
};

// Boundaries that begin and that end a chain.
__global__ void k_chain_flags(const uint32_t *cut, CutArgs a, uint32_t *begin, uint32_t *end) {
  const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (uint64_t)a.nlev * a.nch) return;
  const uint32_t c = (uint32_t)(e % a.nch), v = cut[e];
  begin[e] = v != 0u && !(c > 0u && cut[e - 1] == v);
  end[e] = v != 0u && !(c + 1u < a.nch && cut[e + 1] == v);
}

// The k-th beginning and the k-th end belong to chain k.
__global__ void k_chain_bounds(const uint32_t *cut, CutArgs a, const uint32_t *begin, const uint32_t *end,
                               const uint32_t *at, uint32_t nchains, uint32_t *chain) {
  const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (uint64_t)a.nlev * a.nch) return;
  const uint32_t c = (uint32_t)(e % a.nch), k = (uint32_t)(e / a.nch);
  if (begin[e]) {
    uint32_t *o = chain + (size_t)at[e] * kChainWords;
    o[0] = (uint32_t)a.level_of[k];
    o[1] = cut[e] - 1u;
    o[2] = k;
    o[3] = c;
  }
  if (end[e]) chain[(size_t)(at[(uint64_t)a.nlev * a.nch + e] - nchains) * kChainWords + 4] = c;
}

__global__ void k_chain_sizes(uint32_t *chain, uint32_t n, uint32_t *sizes) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0u) sizes[2 * (size_t)n] = 0u;
  if (i >= n) return;
  uint32_t *o = chain + (size_t)i * kChainWords;
  const uint32_t npart = o[4] - o[3] + 2u, ng = (npart + kGroup - 1) / kGroup;
  o[4] = npart;
  sizes[i] = ng;
  o[7] = sizes[(size_t)n + i] = ng > kMid ? (ng + kMid - 1) / kMid : 0u;
}

// One warp per chain: its first group and group of groups, and the chain of
// its groups.
__global__ void k_chain_groups_of(uint32_t *chain, uint32_t n, const uint32_t *first, uint32_t ngroups,
                                  uint32_t *group_chain) {
  const uint32_t i = (uint32_t)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (i >= n) return;
  uint32_t *o = chain + (size_t)i * kChainWords;
  const uint32_t ng = (o[4] + kGroup - 1) / kGroup;
  if (lane == 0) {
    o[5] = first[i];
    o[6] = first[(size_t)n + i] - ngroups;
  }
  for (uint32_t g = lane; g < ng; g += 32) group_chain[first[i] + g] = i;
}

template <typename T>
struct SumArgs {
  const T *span;
  int nlev, ldr, R;
  const uint32_t *chain, *group_chain;
  uint32_t ngroups, nmids;
  double *gsum, *msum;
  uint32_t *arrived;
  SpanTarget to;
};

// Four columns of a row, FP32 or FP64, from L2: other SMs wrote it.
__device__ __forceinline__ void ld4(const float *p, double (&v)[4]) {
  const float4 f = __ldcg(reinterpret_cast<const float4 *>(p));
  v[0] = f.x;
  v[1] = f.y;
  v[2] = f.z;
  v[3] = f.w;
}
__device__ __forceinline__ void ld4(const double *p, double (&v)[4]) {
  const double2 a = __ldcg(reinterpret_cast<const double2 *>(p));
  const double2 b = __ldcg(reinterpret_cast<const double2 *>(p) + 1);
  v[0] = a.x;
  v[1] = a.y;
  v[2] = b.x;
  v[3] = b.y;
}

// Rows row(0) .. row(n - 1) added in order, eight loads in flight. WIDE: the
// walkers of the warp take a run of the rows each and their sums are added
// pair by pair, so every lane ends with the total (an order of its own, fixed
// as well).
template <int L, bool WIDE, typename F>
__device__ __forceinline__ void add_rows(uint32_t n, F &&row, double (&acc)[4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] = 0.0;
  if constexpr (WIDE && L < 32) {
    const uint32_t wk = (threadIdx.x & 31) / L, share = (n + 32 / L - 1) / (32 / L);
    const uint32_t b = min(n, wk * share), e = min(n, b + share);
    if (b < e) add_rows<L, false>(e - b, [&](uint32_t k) { return row(b + k); }, acc);
    __syncwarp();
#pragma unroll
    for (int o = L; o < 32; o <<= 1)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] += __shfl_xor_sync(~0u, acc[i], o);
    return;
  }
  // (loads past the end repeat the last row, so that no branch parts them)
  for (uint32_t k = 0; k < n; k += 8) {
    double v[8][4];
#pragma unroll
    for (int q = 0; q < 8; ++q) ld4(row(min(k + q, n - 1u)), v[q]);
#pragma unroll
    for (int q = 0; q < 8; ++q)
#pragma unroll
      for (int i = 0; i < 4; ++i) acc[i] += k + q < n ? v[q][i] : 0.0;
  }
}

// One walker (L lanes, four columns each) per group of partials, which it
// adds in chunk order; the one that finishes the last group under a group of
// groups adds those in order, and the one that finishes a chain's last child
// adds the chain. No walker waits, and the order of every sum is the tree's,
// whoever computes it. Most chains are one group: they end without an
// arrival, whose memory ordering costs more than the loads it saves.
//
// WIDE: the whole warp takes one group.
//
// What bounds it: the latency of its dependent loads; one launch in the place
// of two or three.
template <int L, bool WIDE, typename T>
__global__ void __launch_bounds__(128) k_span_sums(const __grid_constant__ SumArgs<T> a) {
  constexpr int Q = WIDE ? 32 : L;  // lanes per group
  const uint32_t g = (blockIdx.x * 128u + threadIdx.x) / Q;
  const int lane = threadIdx.x & 31, col = 4 * (lane % L);
  const uint32_t mask = Q == 32 ? ~0u : ((1u << (L & 31)) - 1u) << (lane / L * L);
  if (g >= a.ngroups) return;
  const bool act = col < a.R && lane % Q < L;
  const uint32_t ci = a.group_chain[g];
  const uint4 c0 = *reinterpret_cast<const uint4 *>(a.chain + (size_t)ci * kChainWords);
  const uint4 c1 = *reinterpret_cast<const uint4 *>(a.chain + (size_t)ci * kChainWords + 4);
  const uint32_t level = c0.x, node = c0.y, first = c0.w, npart = c1.x, g0 = c1.y, m0 = c1.z, nm = c1.w;
  const uint32_t ng = (npart + kGroup - 1) / kGroup, k0 = (g - g0) * kGroup;
  const int lcol = col < a.R ? col : 0;
  double acc[4];
  add_rows<L, WIDE>(min(npart - k0, kGroup), [&](uint32_t k) {
    // the last partial is the head of the last boundary's chunk, the others
    // are the tails of the chunks before it
    k += k0;
    const uint32_t head = k + 1u == npart;
    return a.span + (((size_t)(first - 1u + k) * a.nlev + c0.z) * 2 + (1u - head)) * a.ldr + lcol;
  }, acc);
  auto store = [&](double *p) {
    if (!act) return;
    __stcg(reinterpret_cast<double2 *>(p + col), make_double2(acc[0], acc[1]));
    __stcg(reinterpret_cast<double2 *>(p + col) + 1, make_double2(acc[2], acc[3]));
  };
  // whether these lanes are the last of `children` to arrive (the count then
  // starts over): their rows are released, the others' acquired
  auto last = [&](uint32_t *count, uint32_t children) {
    __syncwarp(mask);
    uint32_t n = 0;
    if (lane % Q == 0) {
      asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(n) : "l"(count) : "memory");
      if (n + 1u == children) *count = 0u;
    }
    n = __shfl_sync(mask, n, 0, Q);
    __syncwarp(mask);  // the first lane's acquire holds for all (a shuffle orders nothing)
    return n + 1u == children;
  };
  if (ng > 1u) {
    store(a.gsum + (size_t)g * a.ldr);
    const double *rows = a.gsum + (size_t)g0 * a.ldr;
    uint32_t n = ng;
    if (nm != 0u) {
      const uint32_t mi = (g - g0) / kMid, b = mi * kMid, children = min(kMid, ng - b);
      if (!last(a.arrived + m0 + mi, children)) return;
      add_rows<L, WIDE>(children, [&](uint32_t k) { return rows + (size_t)(b + k) * a.ldr + lcol; }, acc);
      store(a.msum + (size_t)(m0 + mi) * a.ldr);
      rows = a.msum + (size_t)m0 * a.ldr;
      n = nm;
    }
    if (!last(a.arrived + a.nmids + ci, n)) return;
    add_rows<L, WIDE>(n, [&](uint32_t k) { return rows + (size_t)k * a.ldr + lcol; }, acc);
  }
  if (!act) return;
  if (a.to.store[level])
    *reinterpret_cast<float4 *>(a.to.store[level] + (size_t)node * a.ldr + col) =
        make_float4((float)acc[0], (float)acc[1], (float)acc[2], (float)acc[3]);
  if (level == 0 && a.to.out) store(a.to.out + (size_t)(a.to.out_ids ? a.to.out_ids[node] : node) * a.ldr);
}

unsigned blocks_of(uint64_t n) { return (unsigned)((n + 255) / 256); }

uint32_t to_host(const uint32_t *p, cudaStream_t s) {
  uint32_t v = 0;
  ADATM_CUDA(cudaMemcpyAsync(&v, p, sizeof(v), cudaMemcpyDeviceToHost, s));
  ADATM_CUDA(cudaStreamSynchronize(s));
  return v;
}

}  // namespace

void span_prepare(SpanSums &s, const uint32_t *cut, int nlev, const int *level_of, uint32_t nch, int ldr,
                  cudaStream_t stream) {
  s.nchains = s.ngroups = s.nmids = 0;
  const uint64_t n = (uint64_t)nlev * nch;
  if (n == 0) return;
  CutArgs a;
  a.nlev = nlev;
  a.nch = nch;
  for (int k = 0; k < kMaxModes; ++k) a.level_of[k] = k < nlev ? level_of[k] : 0;
  // flags of the beginnings, then of the ends, in one scan: the chain that
  // ends at a boundary is the number of ends before it
  DevBuf<uint32_t> flags(2 * n, stream), at(2 * n, stream), tmp(scan_tmp_words(2 * n), stream);
  uint32_t *begin = flags.get(), *end = begin + n;
  k_chain_flags<<<blocks_of(n), 256, 0, stream>>>(cut, a, begin, end);
  ADATM_LAUNCH();
  exclusive_scan_u32(begin, at.get(), 2 * n, tmp.get(), stream);
  const uint32_t nc = to_host(at.get() + n, stream);
  if (nc == 0) return;
  s.chain.alloc((size_t)nc * kChainWords, stream);
  k_chain_bounds<<<blocks_of(n), 256, 0, stream>>>(cut, a, begin, end, at.get(), nc, s.chain.get());
  ADATM_LAUNCH();
  // groups, then groups of groups, of every chain, and a last 0
  DevBuf<uint32_t> sizes(2 * (size_t)nc + 1, stream), first(2 * (size_t)nc + 1, stream),
      tmp2(scan_tmp_words(2 * (size_t)nc + 1), stream);
  k_chain_sizes<<<blocks_of(nc), 256, 0, stream>>>(s.chain.get(), nc, sizes.get());
  ADATM_LAUNCH();
  exclusive_scan_u32(sizes.get(), first.get(), 2 * (size_t)nc + 1, tmp2.get(), stream);
  ADATM_CUDA(cudaMemcpyAsync(&s.nmids, first.get() + 2 * (size_t)nc, sizeof(uint32_t), cudaMemcpyDeviceToHost,
                             stream));
  s.ngroups = to_host(first.get() + nc, stream);
  s.nmids -= s.ngroups;
  s.nchains = nc;
  s.group_chain.alloc(s.ngroups, stream);
  k_chain_groups_of<<<blocks_of((uint64_t)nc * 32), 256, 0, stream>>>(s.chain.get(), nc, first.get(), s.ngroups,
                                                                      s.group_chain.get());
  ADATM_LAUNCH();
  s.gsum.alloc((size_t)s.ngroups * ldr, stream);
  s.msum.alloc((size_t)s.nmids * ldr, stream);
  s.arrived.alloc((size_t)s.nmids + nc, stream);
  ADATM_CUDA(cudaMemsetAsync(s.arrived.get(), 0, s.arrived.bytes(), stream));
}

template <typename T>
void span_launch(const SpanSums &s, const T *span, int nlev, int R, int ldr, const SpanTarget &t,
                 cudaStream_t stream) {
  if (s.nchains == 0) return;
  SumArgs<T> a;
  a.span = span;
  a.nlev = nlev;
  a.ldr = ldr;
  a.R = R;
  a.chain = s.chain.get();
  a.group_chain = s.group_chain.get();
  a.ngroups = s.ngroups;
  a.nmids = s.nmids;
  a.gsum = s.gsum.get();
  a.msum = s.msum.get();
  a.arrived = s.arrived.get();
  a.to = t;
  // Few groups (at most one warp each on a full device) are spread over their
  // warps, where a walker alone would add up to 64 rows in eight rounds of
  // loads; many are packed, since most have two or three rows. Measured:
  // 1000 groups of 33 rows, R = 16, 18.7 us packed and 7.5 wide; one root
  // slice of 5000 rows among short ones, R = 16, 18 and 7.4; the 77.9M-nonzero
  // tensor's cuts, R = 32, 51 packed (103 in three launches before).
  auto go = [&](auto lanes) {
    constexpr int L = decltype(lanes)::value;
    if (s.ngroups <= kWideGroups)
      k_span_sums<L, true, T><<<(s.ngroups + 3) / 4, 128, 0, stream>>>(a);
    else
      k_span_sums<L, false, T><<<(unsigned)(((uint64_t)s.ngroups * L + 127) / 128), 128, 0, stream>>>(a);
  };
  if (R <= 16) go(std::integral_constant<int, 4>{});
  else if (R <= 32) go(std::integral_constant<int, 8>{});
  else if (R <= 64) go(std::integral_constant<int, 16>{});
  else go(std::integral_constant<int, 32>{});
  ADATM_LAUNCH();
}

template void span_launch<float>(const SpanSums &, const float *, int, int, int, const SpanTarget &,
                                 cudaStream_t);
template void span_launch<double>(const SpanSums &, const double *, int, int, int, const SpanTarget &,
                                  cudaStream_t);

}  // namespace adatm
