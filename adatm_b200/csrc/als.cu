// als.cu -- dense CP-ALS kernels (see als.cuh).
#include <algorithm>
#include <mutex>

#include "als.cuh"

namespace adatm {

namespace {
void set_attributes();
}

void AlsWork::init(int nmodes_, int R_, int nblocks_, int max_iters, cudaStream_t s) {
  nmodes = nmodes_;
  R = R_;
  ldr = ldr_of(R_);
  nblocks = nblocks_;
  vinv64.alloc((size_t)R * R, s);
  part_gram.alloc((size_t)nblocks * R * R, s);
  part_max.alloc((size_t)nblocks * R, s);
  part_inner.alloc((size_t)nblocks * R, s);
  lambda.alloc(R, s);
  scalars.alloc(8, s);
  iter.alloc(1, s);
  arrived.alloc(1, s);
  ADATM_CUDA(cudaMemsetAsync(arrived.get(), 0, sizeof(uint32_t), s));
  max_trace = std::max(1, max_iters);
  fit_trace.alloc(max_trace, s);
  ADATM_CUDA(cudaMemsetAsync(scalars.get(), 0, 8 * sizeof(double), s));
  ADATM_CUDA(cudaMemsetAsync(iter.get(), 0, sizeof(int), s));
  ADATM_CUDA(cudaMemsetAsync(fit_trace.get(), 0, max_trace * sizeof(double), s));
  set_attributes();
}

namespace {

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void k_factor_init(float *A, __nv_bfloat16 *Ab, uint64_t rows, int R, int ldr,
                              uint64_t key) {
  const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= rows * (uint64_t)ldr) return;
  const uint64_t i = e / ldr;
  const int r = (int)(e % ldr);
  float v = 0.f;
  if (r < R) {
    const uint64_t x = i * (uint64_t)R + r;
    v = (float)((double)(mix64(key + x) >> 11) * (1.0 / 9007199254740992.0));
  }
  if (Ab) {
    // BF16 factors: the rounded value is the factor (see to_bf16)
    const __nv_bfloat16 b = __float2bfloat16(v);
    Ab[e] = b;
    v = __bfloat162float(b);
  }
  A[e] = v;
}

__global__ void k_to_bf16(float *A, __nv_bfloat16 *Ab, uint64_t n) {
  const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < n) {
    const __nv_bfloat16 b = __float2bfloat16(A[e]);
    Ab[e] = b;
    A[e] = __bfloat162float(b);
  }
}

constexpr int kFrobThreads = 256;

__global__ void k_frob_partial(const double *v, uint64_t n, double *part) {
  double s = 0;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    s += v[i] * v[i];
  __shared__ double red[kFrobThreads];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = kFrobThreads / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = red[0];
}

__global__ void k_frob_final(const double *part, int n, double *out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0;
    for (int i = 0; i < n; ++i) s += part[i];
    out[0] = s;
  }
}

// ---------------------------------------------------------------------------
// Gram Hadamard + inverse, one block. V = Hadamard of every G[m], m != mode,
// is symmetric positive definite, so Gauss-Jordan elimination in place needs
// no pivoting (each pivot is a diagonal entry of a Schur complement of V,
// hence positive).
//
// V stays in registers: warp w holds rows w * RW .. (RW = RMAX / WARPS), lane l the
// columns l, l + 32, ... Per step the pivot row goes through shared memory
// (two buffers, one barrier) and the pivot column's entries of a warp's own
// rows through shuffles. What bounds it: the latency of R dependent steps
// (barrier, division, multiply-add), which is why a step does nothing else.
// Eight warps; sixteen above R = 64, where eight would hold 64 doubles a
// thread (470 us at R = 128), while at R = 64 they are slower (34 us for 31).
// Measured before (V in shared memory, three barriers per step) and now, us:
// R=8 6.9 -> 6.2, R=16 10.2 -> 9.2, R=24 20 -> 12.3, R=32 30 -> 9.8,
// R=48 72 -> 32, R=64 146 -> 31, R=100 481 -> 304, R=128 951 -> 367.
// ---------------------------------------------------------------------------
template <int RMAX, int WARPS>
__global__ void __launch_bounds__(32 * WARPS)
    k_gram_inverse(const __grid_constant__ GramSet g, int nmodes, int mode, int R, double *X) {
  constexpr int RW = RMAX / WARPS, C = (RMAX + 31) / 32;
  extern __shared__ double rows[];  // two pivot rows, then V (R x R) before and after
  double *V = rows + 64 * C;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int U = RMAX >= 32 ? 4 : 1;
  for (int e0 = threadIdx.x; e0 < R * R; e0 += 32 * WARPS * U) {
    double h[U];
#pragma unroll
    for (int u = 0; u < U; ++u) h[u] = 1.0;
    for (int m = 0; m < nmodes; ++m) {
      if (m == mode) continue;
#pragma unroll
      for (int u = 0; u < U; ++u) h[u] *= g.G[m][min(e0 + 32 * WARPS * u, R * R - 1)];
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (e0 + 32 * WARPS * u < R * R) V[e0 + 32 * WARPS * u] = h[u];
  }
  __syncthreads();
  double v[RW][C];
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int i = warp * RW + r, k = lane + 32 * c;
      v[r][c] = i < R && k < R ? V[i * R + k] : 0.0;
    }
  for (int w = 0; w < WARPS; ++w) {
#pragma unroll
    for (int rr = 0; rr < RW; ++rr) {
      const int j = w * RW + rr;
      if (j >= R) break;
      double *row = rows + (j & 1) * 32 * C;
      if (warp == w) {
#pragma unroll
        for (int c = 0; c < C; ++c) row[lane + 32 * c] = v[rr][c];
      }
      __syncthreads();
      const double p = row[j];
      // pivot row: V[j][k] = (k == j ? 1 : V[j][k]) / p
      double q[C];
#pragma unroll
      for (int c = 0; c < C; ++c) q[c] = (lane + 32 * c == j ? 1.0 : row[lane + 32 * c]) / p;
      // other rows: V[i][k] = (k == j ? 0 : V[i][k]) - V[i][j] * V[j][k]
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        double f = v[r][0];
#pragma unroll
        for (int c = 1; c < C; ++c) f = (j >> 5) == c ? v[r][c] : f;
        f = __shfl_sync(~0u, f, j & 31);
        if (warp == w && r == rr) {
#pragma unroll
          for (int c = 0; c < C; ++c) v[r][c] = q[c];
        } else {
#pragma unroll
          for (int c = 0; c < C; ++c) v[r][c] = (lane + 32 * c == j ? 0.0 : v[r][c]) - f * q[c];
        }
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const int i = warp * RW + r, k = lane + 32 * c;
      if (i < R && k < R) V[i * R + k] = v[r][c];
    }
  __syncthreads();
  for (int e = threadIdx.x; e < R * R; e += 32 * WARPS) {
    // symmetrise: the two triangles differ only by rounding
    const int i = e / R, k = e % R;
    X[e] = 0.5 * (V[e] + V[k * R + i]);
  }
}

template <int RMAX>
constexpr size_t inverse_smem(int R) {
  const int C = (RMAX + 31) / 32;
  return sizeof(double) * (size_t)(R * R + 64 * C);
}

// ---------------------------------------------------------------------------
// Row update A_raw = M * Vinv (or A_raw = M when vinv == nullptr), with
// per-block FP64 partial Gram and column maxima of A_raw; then what follows
// from the partials of all blocks: lambda, the Gram, the normalised rows, the
// fit.
// ---------------------------------------------------------------------------
struct FinishArgs {
  const double *part_gram, *part_max;  // per block of the update
  int nblocks, R, ldr;
  double *G;                    // R x R
  double *lam;                  // nullptr: only the Gram is wanted
  const int *iter;
  // rows scaled by 1 / lambda
  float *A;
  __nv_bfloat16 *Ab;
  uint64_t rows;
  // <A, M> per column (M != nullptr) and the fit (fit != 0)
  const double *M;
  double *part_inner;
  int fit;
  GramSet g;
  int nmodes;
  double *scalars, *trace;
  int max_trace;
  int *iter_out;
  uint32_t *arrived;            // blocks done, 0 between launches
};

struct UpdArgs {
  int split;           // Gram products as 3 TF32 terms (FP32 rows) or 1 (BF16-valued rows)
  const double *Md;    // MTTKRP rows (FP64) of an update, or nullptr
  const float *M;      // rows whose Gram alone is wanted (vinv == nullptr)
  const double *vinv;  // R x R fp64, or nullptr for identity
  float *A;           // output rows (may alias M when vinv == nullptr)
  uint64_t rows;
  int R, ldr;
  double *part_gram;  // gridDim x R x R
  double *part_max;   // gridDim x R
  int last_finishes;  // the last block goes on with `fin`
  FinishArgs fin;
};

// Whether this block is the last of `blocks` to get here (the count then
// starts over). What the others wrote before is visible to all its threads,
// which read it through L2. No block waits.
__device__ __forceinline__ bool last_block(uint32_t *count, uint32_t blocks) {
  __shared__ uint32_t s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t n = atomicAdd(count, 1u);
    s_last = n + 1u == blocks;
    if (s_last) *count = 0u;
    __threadfence();
  }
  __syncthreads();
  return s_last != 0u;
}

// lambda (2-norm on the first iteration, max-norm floored at 1 after) from the
// blocks' partials into slam; `red`: 256 doubles.
__device__ __forceinline__ void derive_lambda(const FinishArgs &f, double *slam, double *red) {
  const int tid = threadIdx.x, R = f.R;
  const bool first = f.iter == nullptr || *f.iter == 0;
  const int parts = 256 / R;  // R <= 128
  const int r = tid % R, q = tid / R;
  double v = 0.0;
  if (q < parts) {
    if (first) {
#pragma unroll 8
      for (int b = q; b < f.nblocks; b += parts) v += f.part_gram[(size_t)b * R * R + r * R + r];
    } else {
#pragma unroll 8
      for (int b = q; b < f.nblocks; b += parts) v = fmax(v, f.part_max[(size_t)b * R + r]);
    }
  }
  red[tid] = v;
  __syncthreads();
  if (tid < R) {
    double a = 0.0;
    for (int k = 0; k < parts; ++k) a = first ? a + red[k * R + tid] : fmax(a, red[k * R + tid]);
    slam[tid] = first ? sqrt(a) : fmax(a, 1.0);
  }
  __syncthreads();
}

// Entries [32 c, 32 c + 32) of the Gram: the block's warps split the partials,
// so that no thread walks a long chain of dependent L2 loads.
constexpr int kFinEntries = 32;
constexpr int kFinParts = 256 / kFinEntries;
__device__ __forceinline__ void gram_entries(const FinishArgs &f, int c, const double *slam, double *red) {
  const int tid = threadIdx.x, R = f.R;
  const int e = c * kFinEntries + tid % kFinEntries, q = tid / kFinEntries;
  double acc = 0.0;
  if (e < R * R)
#pragma unroll 8
    for (int b = q; b < f.nblocks; b += kFinParts) acc += f.part_gram[(size_t)b * R * R + e];
  red[tid] = acc;
  __syncthreads();
  if (tid < kFinEntries && e < R * R) {
    double sum = 0.0;
    for (int k = 0; k < kFinParts; ++k) sum += red[k * kFinEntries + tid];
    if (f.lam) sum /= slam[e / R] * slam[e % R];
    f.G[e] = sum;
  }
  __syncthreads();
}

__host__ __device__ constexpr int finalize_blocks(int R) { return (R * R + kFinEntries - 1) / kFinEntries; }

// A /= lambda (fp32), bf16 copy, optional partial <A, M> per column into
// part_inner[block]: rows block * GROUPS .. in steps of blocks * GROUPS. `red`:
// 1024 doubles.
template <int LANES>
__device__ __forceinline__ void scale_rows(const FinishArgs &f, const double *lam, uint64_t block,
                                           uint64_t blocks, double *red) {
  constexpr int GROUPS = 256 / LANES;
  const int tid = threadIdx.x, R = f.R, ldr = f.ldr;
  const int g = tid / LANES, t = tid % LANES, col = 4 * t;
  const bool act = col < R;
  float4 il = make_float4(0.f, 0.f, 0.f, 0.f);
  if (act) {
    il.x = col + 0 < R ? (float)(1.0 / lam[col + 0]) : 0.f;
    il.y = col + 1 < R ? (float)(1.0 / lam[col + 1]) : 0.f;
    il.z = col + 2 < R ? (float)(1.0 / lam[col + 2]) : 0.f;
    il.w = col + 3 < R ? (float)(1.0 / lam[col + 3]) : 0.f;
  }
  double in0 = 0, in1 = 0, in2 = 0, in3 = 0;
  for (uint64_t i = block * GROUPS + g; i < f.rows; i += blocks * GROUPS) {
    if (!act) continue;
    float4 v = __ldcg(reinterpret_cast<float4 *>(f.A + i * ldr + col));
    v.x *= il.x;
    v.y *= il.y;
    v.z *= il.z;
    v.w *= il.w;
    if (f.Ab) {
      // BF16 factors: the rounded row replaces the FP32 row too, so the
      // Gram, the MTTKRPs and the fit all see the same factor
      __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y);
      __nv_bfloat162 hi = __floats2bfloat162_rn(v.z, v.w);
      uint2 raw;
      raw.x = *reinterpret_cast<uint32_t *>(&lo);
      raw.y = *reinterpret_cast<uint32_t *>(&hi);
      *reinterpret_cast<uint2 *>(f.Ab + i * ldr + col) = raw;
      const float2 flo = __bfloat1622float2(lo), fhi = __bfloat1622float2(hi);
      v = make_float4(flo.x, flo.y, fhi.x, fhi.y);
    }
    *reinterpret_cast<float4 *>(f.A + i * ldr + col) = v;
    if (f.M) {
      const double2 lo = *reinterpret_cast<const double2 *>(f.M + i * ldr + col);
      const double2 hi = *reinterpret_cast<const double2 *>(f.M + i * ldr + col + 2);
      in0 += (double)v.x * lo.x;
      in1 += (double)v.y * lo.y;
      in2 += (double)v.z * hi.x;
      in3 += (double)v.w * hi.y;
    }
  }
  if (f.M) {
    red[tid * 4 + 0] = in0;
    red[tid * 4 + 1] = in1;
    red[tid * 4 + 2] = in2;
    red[tid * 4 + 3] = in3;
    __syncthreads();
    if (tid < 4 * LANES) {
      const int tt = tid / 4, c = tid % 4;
      double s = 0;
      for (int gi = 0; gi < GROUPS; ++gi) s += red[(gi * LANES + tt) * 4 + c];
      const int column = 4 * tt + c;
      if (column < R) f.part_inner[block * R + column] = s;
    }
    __syncthreads();
  }
}

// fit = 1 - sqrt(||X||^2 + ||Z||^2 - 2 <X, Z>) / ||X||; one block. `red`: 256
// doubles.
__device__ __forceinline__ void fit_step(const GramSet &g, int nmodes, int R, const double *lam,
                                         const double *part_inner, int nblocks, double *scalars, double *trace,
                                         int max_trace, int *iter, double *red) {
  const int tid = threadIdx.x;
  double nrm = 0;
  constexpr int U = 4;  // entries whose loads are in flight together
  for (int e0 = tid; e0 < R * R; e0 += U * 256) {
    double h[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = min(e0 + 256 * u, R * R - 1);
      h[u] = lam[e / R] * lam[e % R];
    }
    for (int m = 0; m < nmodes; ++m) {
      const double *G = g.G[m];
#pragma unroll
      for (int u = 0; u < U; ++u) h[u] *= __ldcg(G + min(e0 + 256 * u, R * R - 1));
    }
#pragma unroll
    for (int u = 0; u < U; ++u) nrm += e0 + 256 * u < R * R ? h[u] : 0.0;
  }
  // <X, Z> = sum_r lam_r sum_b part_inner[b][r]: 256 / R threads per column
  double inner = 0;
  {
    const int parts = 256 / R, r = tid % R, q = tid / R;
    if (q < parts) {
#pragma unroll 8
      for (int b = q; b < nblocks; b += parts) inner += __ldcg(part_inner + (size_t)b * R + r);
      inner *= lam[r];
    }
  }
  red[tid] = nrm;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (tid < o) red[tid] += red[tid + o];
    __syncthreads();
  }
  const double norm = fabs(red[0]);
  __syncthreads();
  red[tid] = inner;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (tid < o) red[tid] += red[tid + o];
    __syncthreads();
  }
  if (tid == 0) {
    const double in = red[0];
    const double ttn = scalars[0];
    const double fit = 1.0 - sqrt(ttn + norm - 2.0 * in) / sqrt(ttn);
    scalars[1] = fit;
    scalars[2] = norm;
    scalars[3] = in;
    const int it = *iter;
    if (it < max_trace) trace[it] = fit;
    *iter = it + 1;
  }
}

// All of what follows an update of few row groups, by one block. `sums`: R * R
// doubles, `red`: 1024.
template <int LANES>
__device__ __forceinline__ void finish_alone(const FinishArgs &f, double *sums, double *slam, double *red) {
  const int tid = threadIdx.x, R = f.R;
  constexpr int U = 4;  // entries whose loads are in flight together
  for (int e0 = tid; e0 < R * R; e0 += U * 256) {
    double acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u) acc[u] = 0.0;
    for (int b = 0; b < f.nblocks; ++b)
#pragma unroll
      for (int u = 0; u < U; ++u)
        acc[u] += __ldcg(f.part_gram + (size_t)b * R * R + min(e0 + 256 * u, R * R - 1));
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = e0 + 256 * u;
      if (e >= R * R) break;
      sums[e] = acc[u];
      if (!f.lam) f.G[e] = acc[u];
    }
  }
  if (!f.lam) return;
  __syncthreads();
  if (tid < R) {
    double l = 1.0;
    if (*f.iter == 0) {
      l = sqrt(sums[tid * R + tid]);
    } else {
      for (int b = 0; b < f.nblocks; ++b) l = fmax(l, __ldcg(f.part_max + (size_t)b * R + tid));
    }
    slam[tid] = l;
    f.lam[tid] = l;
  }
  __syncthreads();
  for (int e = tid; e < R * R; e += 256) f.G[e] = sums[e] / (slam[e / R] * slam[e % R]);
  scale_rows<LANES>(f, slam, 0, 1, red);
  if (f.fit) {
    __threadfence();
    __syncthreads();
    fit_step(f.g, f.nmodes, R, slam, f.part_inner, 1, f.scalars, f.trace, f.max_trace, f.iter_out, red);
  }
}

// The same by a grid, ranks up to 32: every block derives lambda, scales its
// rows and takes its share of the Gram; the last one to end computes the fit.
template <int LANES>
__global__ void __launch_bounds__(256) k_finish(const __grid_constant__ FinishArgs f) {
  __shared__ double slam[128];
  __shared__ double red[1024];
  derive_lambda(f, slam, red);
  if (blockIdx.x == 0 && (int)threadIdx.x < f.R) f.lam[threadIdx.x] = slam[threadIdx.x];
  const int chunks = finalize_blocks(f.R);
  for (int c = blockIdx.x; c < chunks; c += gridDim.x) gram_entries(f, c, slam, red);
  scale_rows<LANES>(f, slam, blockIdx.x, gridDim.x, red);
  if (f.fit && last_block(f.arrived, gridDim.x))
    fit_step(f.g, f.nmodes, f.R, slam, f.part_inner, (int)gridDim.x, f.scalars, f.trace, f.max_trace,
             f.iter_out, red);
}

// Larger ranks in two launches: lambda and the Gram (or the Gram alone), then
// the rows and the fit.
__global__ void __launch_bounds__(256) k_finalize(const __grid_constant__ FinishArgs f) {
  __shared__ double slam[128];
  __shared__ double red[256];
  if (f.lam) {
    derive_lambda(f, slam, red);
    if (blockIdx.x == 0 && (int)threadIdx.x < f.R) f.lam[threadIdx.x] = slam[threadIdx.x];
  }
  gram_entries(f, blockIdx.x, slam, red);
}

template <int LANES>
__global__ void __launch_bounds__(256) k_scale(const __grid_constant__ FinishArgs f) {
  __shared__ double red[1024];
  scale_rows<LANES>(f, f.lam, blockIdx.x, gridDim.x, red);
  if (f.fit && last_block(f.arrived, gridDim.x))
    fit_step(f.g, f.nmodes, f.R, f.lam, f.part_inner, (int)gridDim.x, f.scalars, f.trace, f.max_trace,
             f.iter_out, red);
}

// One m16n8k8 TF32 tensor-core product with FP32 accumulation, c += a * b
// (A 16 x 8 row-major, B 8 x 8 column-major, per-thread fragments of the
// warp-wide tiles).
__device__ __forceinline__ void mma_tf32(float c[4], const uint32_t a[4], const uint32_t b[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;\n" : "=r"(r) : "f"(x));
  return r;
}

// Row pass of a mode update (or of a plain Gram). Each block takes row
// groups of 256 / LANES rows; the rows (A = M V^-1, or M itself) are staged
// in shared memory and their Gram X^T X is taken on the tensor cores: G is
// tiled in 16 x 8 tiles spread over the block's 8 warps; every 8 rows of a
// tile are one m16n8k8 TF32 MMA step with FP32 accumulation, added to FP64
// per-thread sums after the step. FP32 rows split into a TF32 big
// part and a TF32 remainder, and big*big + big*rem + rem*big keeps the
// products to ~2^-22 (split = 1); BF16-valued rows are exact in TF32 and
// take one product.
template <int LANES>
__global__ void __launch_bounds__(256) k_update(const __grid_constant__ UpdArgs a) {
  constexpr int GROUPS = 256 / LANES;
  constexpr int RMAX = 4 * LANES;
  constexpr int RS = RMAX + 8;          // staged row stride (bank-conflict free MMA loads)
  constexpr int TN = RMAX / 8;          // 8-column tiles of G
  constexpr int NT = (RMAX / 16) * TN;  // 16 x 8 tiles
  constexpr int TPW = (NT + 7) / 8;     // tiles per warp
  extern __shared__ double usm[];
  double *vinv = usm;                                            // RMAX x RMAX
  float *rowbuf = reinterpret_cast<float *>(usm + RMAX * RMAX);  // GROUPS x RS
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, gid = lane >> 2, tig = lane & 3;
  const int g = tid / LANES, t = tid % LANES, col = 4 * t;
  const int R = a.R;
  const bool act = col < R;
  const unsigned gmask =
      LANES == 32 ? 0xffffffffu : (((1u << LANES) - 1u) << ((tid & 31) / LANES * LANES));
  if (a.vinv) {
    for (int e = tid; e < RMAX * RMAX; e += 256) {
      const int k = e / RMAX, c = e % RMAX;
      vinv[e] = (k < R && c < R) ? a.vinv[k * R + c] : 0.0;
    }
  }
  double gacc[TPW][4];
#pragma unroll
  for (int tt = 0; tt < TPW; ++tt)
#pragma unroll
    for (int q = 0; q < 4; ++q) gacc[tt][q] = 0.0;
  double cmax = 0.0;
  __syncthreads();
  const int kq = (R + 3) / 4;
  for (uint64_t row0 = (uint64_t)blockIdx.x * GROUPS; row0 < a.rows;
       row0 += (uint64_t)gridDim.x * GROUPS) {
    const uint64_t i = row0 + g;
    const bool valid = i < a.rows;
    double md[4] = {0.0, 0.0, 0.0, 0.0};
    if (valid && act) {
      if (a.Md) {
        const double2 lo = *reinterpret_cast<const double2 *>(a.Md + i * a.ldr + col);
        const double2 hi = *reinterpret_cast<const double2 *>(a.Md + i * a.ldr + col + 2);
        md[0] = lo.x;
        md[1] = lo.y;
        md[2] = hi.x;
        md[3] = hi.y;
      } else {
        const float4 f = *reinterpret_cast<const float4 *>(a.M + i * a.ldr + col);
        md[0] = f.x;
        md[1] = f.y;
        md[2] = f.z;
        md[3] = f.w;
      }
    }
    float4 o;
    if (a.vinv) {
      // A = M V^-1 with V^-1 and the sums in FP64: V (the Hadamard of the
      // other modes' Grams) is often ill-conditioned, and FP32 sums of its
      // inverse's large entries of both signs lose the fit's digits
      double o0 = 0.0, o1 = 0.0, o2 = 0.0, o3 = 0.0;
      for (int kk = 0; kk < kq; ++kk) {
        const double m4[4] = {__shfl_sync(gmask, md[0], kk, LANES), __shfl_sync(gmask, md[1], kk, LANES),
                              __shfl_sync(gmask, md[2], kk, LANES), __shfl_sync(gmask, md[3], kk, LANES)};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const double *vr = vinv + (4 * kk + q) * RMAX + col;
          const double2 lo = *reinterpret_cast<const double2 *>(vr);
          const double2 hi = *reinterpret_cast<const double2 *>(vr + 2);
          o0 = fma(m4[q], lo.x, o0);
          o1 = fma(m4[q], lo.y, o1);
          o2 = fma(m4[q], hi.x, o2);
          o3 = fma(m4[q], hi.y, o3);
        }
      }
      o = make_float4((float)o0, (float)o1, (float)o2, (float)o3);
      if (valid && act) *reinterpret_cast<float4 *>(a.A + i * a.ldr + col) = o;
    } else {
      o = make_float4((float)md[0], (float)md[1], (float)md[2], (float)md[3]);
    }
    *reinterpret_cast<float4 *>(rowbuf + g * RS + col) =
        valid ? o : make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
#pragma unroll
    for (int tt = 0; tt < TPW; ++tt) {
      const int tile = warp + 8 * tt;
      const int i0 = (tile / TN) * 16, j0 = (tile % TN) * 8;
      if (tile < NT && i0 < R && j0 < R) {
#pragma unroll
        for (int k0 = 0; k0 < GROUPS; k0 += 8) {
          float c[4] = {0.f, 0.f, 0.f, 0.f};
          // A = X^T (rows i0.., the group's rows as k), B = X (columns j0..)
          const float *x0 = rowbuf + (k0 + tig) * RS, *x1 = rowbuf + (k0 + tig + 4) * RS;
          const float av[4] = {x0[i0 + gid], x0[i0 + gid + 8], x1[i0 + gid], x1[i0 + gid + 8]};
          const float bv[2] = {x0[j0 + gid], x1[j0 + gid]};
          uint32_t ab[4], bb[2];
#pragma unroll
          for (int q = 0; q < 4; ++q) ab[q] = to_tf32(av[q]);
          bb[0] = to_tf32(bv[0]);
          bb[1] = to_tf32(bv[1]);
          mma_tf32(c, ab, bb);
          if (a.split) {
            uint32_t as[4], bs[2];
#pragma unroll
            for (int q = 0; q < 4; ++q) as[q] = to_tf32(av[q] - __uint_as_float(ab[q]));
            bs[0] = to_tf32(bv[0] - __uint_as_float(bb[0]));
            bs[1] = to_tf32(bv[1] - __uint_as_float(bb[1]));
            mma_tf32(c, ab, bs);
            mma_tf32(c, as, bb);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) gacc[tt][q] += (double)c[q];
        }
      }
    }
    if (tid < R)
      for (int gi = 0; gi < GROUPS; ++gi) cmax = fmax(cmax, (double)rowbuf[gi * RS + tid]);
    __syncthreads();
  }
#pragma unroll
  for (int tt = 0; tt < TPW; ++tt) {
    const int tile = warp + 8 * tt;
    const int i0 = (tile / TN) * 16, j0 = (tile % TN) * 8;
    if (tile >= NT || i0 >= R || j0 >= R) continue;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = i0 + gid + (q >= 2 ? 8 : 0), j = j0 + 2 * tig + (q & 1);
      if (i < R && j < R) a.part_gram[(size_t)blockIdx.x * R * R + i * R + j] = gacc[tt][q];
    }
  }
  if (tid < R) a.part_max[(size_t)blockIdx.x * R + tid] = cmax;
  if constexpr (LANES < 32) {
    __shared__ double slam[128];
    __shared__ double red[1024];
    if (a.last_finishes && last_block(a.fin.arrived, gridDim.x)) finish_alone<LANES>(a.fin, usm, slam, red);
  }
}

__global__ void __launch_bounds__(256) k_fit(GramSet g, int nmodes, int R, const double *lam,
                                             const double *part_inner, int nblocks, double *scalars,
                                             double *trace, int max_trace, int *iter) {
  __shared__ double red[256];
  fit_step(g, nmodes, R, lam, part_inner, nblocks, scalars, trace, max_trace, iter, red);
}

int lanes_for(int R) {
  if (R <= 16) return 4;
  if (R <= 32) return 8;
  if (R <= 64) return 16;
  if (R <= 128) return 32;
  throw BadInput("rank above 128 is not supported by the GPU kernels");
}

template <int LANES>
constexpr size_t update_smem() {
  return (size_t)(4 * LANES * 4 * LANES) * sizeof(double) +
         (size_t)((256 / LANES) * (4 * LANES + 8)) * sizeof(float);
}

template <int LANES>
void launch_update(const UpdArgs &u, int nblocks, cudaStream_t s) {
  k_update<LANES><<<nblocks, 256, update_smem<LANES>(), s>>>(u);
  ADATM_LAUNCH();
}

// Kernels with more than 48 KB of dynamic shared memory must be opted in
// once, before any stream capture.
void set_attributes() {
  ADATM_CUDA(cudaFuncSetAttribute(k_update<4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)update_smem<4>()));
  ADATM_CUDA(cudaFuncSetAttribute(k_update<8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)update_smem<8>()));
  ADATM_CUDA(cudaFuncSetAttribute(k_update<16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)update_smem<16>()));
  ADATM_CUDA(cudaFuncSetAttribute(k_update<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)update_smem<32>()));
  ADATM_CUDA(cudaFuncSetAttribute((k_gram_inverse<128, 16>), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)inverse_smem<128>(128)));
}

// Row blocks of the update: enough to give every block at least one full
// batch of rows, at most the workspace's partial slots.
int update_blocks(uint64_t rows, int R, int max_blocks) {
  const uint64_t groups = 256 / lanes_for(R);
  const uint64_t need = (rows + groups - 1) / groups;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)max_blocks, need));
}

void run_update(const UpdArgs &u, int nblocks, cudaStream_t s) {
  switch (lanes_for(u.R)) {
    case 4: launch_update<4>(u, nblocks, s); break;
    case 8: launch_update<8>(u, nblocks, s); break;
    case 16: launch_update<16>(u, nblocks, s); break;
    default: launch_update<32>(u, nblocks, s); break;
  }
}

}  // namespace

void factor_init_device(float *A, __nv_bfloat16 *Ab, uint64_t rows, int R, int ldr, uint64_t seed,
                        uint64_t mode, cudaStream_t s) {
  auto hmix = [](uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  };
  const uint64_t key = hmix(seed * 0x100000001B3ull + mode);
  const uint64_t n = rows * (uint64_t)ldr;
  if (n == 0) return;
  k_factor_init<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(A, Ab, rows, R, ldr, key);
  ADATM_LAUNCH();
}

void to_bf16(float *A, __nv_bfloat16 *Ab, uint64_t rows, int ldr, cudaStream_t s) {
  const uint64_t n = rows * (uint64_t)ldr;
  if (n == 0) return;
  k_to_bf16<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(A, Ab, n);
  ADATM_LAUNCH();
}

// Whether the update's last block finishes alone: up to four row groups (one
// block each) and rank 64. A block then takes the partials and rows in a few
// rounds of loads; with more groups, or the larger Grams of more columns, the
// grids below are faster than one block. Measured on 30 rows, us, three
// launches (without the gaps between them) / this: R=16 13.7 / 10.3, R=32
// 17.8 / 13.6, R=48 22.8 / 21.8, R=64 26.1 / 26.8, R=100 32.9 / 43.2.
bool last_finishes(int nblocks, int R) { return nblocks <= 4 && R <= 64; }

// Whether the grid that scales the rows takes lambda and the Gram as well:
// ranks up to 32. Larger Grams have many partials per entry: few blocks sum
// them when the rows are few, and each block takes several rounds when they
// are many. 3000 rows, us, k_finalize + k_scale / one kernel: R=16 7.4 + 4.0 /
// 9.5, R=32 7.8 + 3.4 / 10.5, R=48 23.5 + 4.2 / 31.2, R=100 68.7 + 4.4 / 98
// (the last two with partials read past L1, which neither does any more:
// k_finalize now takes 15.3 and 27.7, where it took 20.1 and 41.8 before).
bool one_finish(int R) { return R <= 32; }

FinishArgs finish_args(const UpdArgs &u, int nblocks, double *G) {
  FinishArgs f = {};
  f.part_gram = u.part_gram;
  f.part_max = u.part_max;
  f.nblocks = nblocks;
  f.R = u.R;
  f.ldr = u.ldr;
  f.G = G;
  return f;
}

void gram(const float *A, uint64_t rows, int R, int ldr, double *G, AlsWork &w, cudaStream_t s,
          bool bf16_rows) {
  UpdArgs u = {};
  u.split = bf16_rows ? 0 : 1;
  u.M = A;
  u.rows = rows;
  u.R = R;
  u.ldr = ldr;
  u.part_gram = w.part_gram.get();
  u.part_max = w.part_max.get();
  const int nb = update_blocks(rows, R, w.nblocks);
  u.fin = finish_args(u, nb, G);
  u.fin.arrived = w.arrived.get();
  u.last_finishes = last_finishes(nb, R);
  run_update(u, nb, s);
  if (u.last_finishes) return;
  k_finalize<<<finalize_blocks(R), 256, 0, s>>>(u.fin);
  ADATM_LAUNCH();
}

void frob_sq(const double *vals, uint64_t n, AlsWork &w, cudaStream_t s) {
  const int blocks = 256;
  if (w.frob_part.n < (size_t)blocks) w.frob_part.alloc(blocks, s);
  k_frob_partial<<<blocks, kFrobThreads, 0, s>>>(vals, n, w.frob_part.get());
  ADATM_LAUNCH();
  k_frob_final<<<1, 32, 0, s>>>(w.frob_part.get(), blocks, w.scalars.get());
  ADATM_LAUNCH();
  ADATM_CUDA(cudaStreamSynchronize(s));
}

void gram_inverse(const GramSet &g, int mode, AlsWork &w, cudaStream_t s) {
  if (w.R <= 16)
    k_gram_inverse<16, 8><<<1, 256, inverse_smem<16>(w.R), s>>>(g, w.nmodes, mode, w.R, w.vinv64.get());
  else if (w.R <= 32)
    k_gram_inverse<32, 8><<<1, 256, inverse_smem<32>(w.R), s>>>(g, w.nmodes, mode, w.R, w.vinv64.get());
  else if (w.R <= 64)
    k_gram_inverse<64, 8><<<1, 256, inverse_smem<64>(w.R), s>>>(g, w.nmodes, mode, w.R, w.vinv64.get());
  else
    k_gram_inverse<128, 16><<<1, 512, inverse_smem<128>(w.R), s>>>(g, w.nmodes, mode, w.R, w.vinv64.get());
  ADATM_LAUNCH();
}

void update_factor(const double *M, uint64_t rows, float *A, __nv_bfloat16 *Ab, double *G_mode,
                   bool inner, const GramSet *fit_grams, AlsWork &w, cudaStream_t s) {
  UpdArgs u = {};
  u.split = 1;
  u.Md = M;
  u.vinv = w.vinv64.get();
  u.A = A;
  u.rows = rows;
  u.R = w.R;
  u.ldr = w.ldr;
  u.part_gram = w.part_gram.get();
  u.part_max = w.part_max.get();
  const int nb = update_blocks(rows, w.R, w.nblocks);
  FinishArgs f = finish_args(u, nb, G_mode);
  f.lam = w.lambda.get();
  f.iter = w.iter.get();
  f.A = A;
  f.Ab = Ab;
  f.rows = rows;
  f.M = inner ? M : nullptr;
  f.part_inner = w.part_inner.get();
  // with BF16 factors the fit waits for the Gram of the rounded rows
  f.fit = inner && fit_grams != nullptr && Ab == nullptr;
  if (fit_grams) f.g = *fit_grams;
  f.nmodes = w.nmodes;
  f.scalars = w.scalars.get();
  f.trace = w.fit_trace.get();
  f.max_trace = w.max_trace;
  f.iter_out = w.iter.get();
  f.arrived = w.arrived.get();
  u.last_finishes = last_finishes(nb, w.R);
  // one block per row group, and where the Gram is taken in the same launch at
  // least one per kFinEntries of its entries
  const bool one = one_finish(w.R);
  const int fb = one ? std::min(w.nblocks, std::max(nb, finalize_blocks(w.R))) : nb;
  if (inner) w.inner_blocks = u.last_finishes ? 1 : fb;
  u.fin = f;
  run_update(u, nb, s);
  if (!u.last_finishes) {
    if (!one) {
      k_finalize<<<finalize_blocks(w.R), 256, 0, s>>>(f);
      ADATM_LAUNCH();
    }
    switch (lanes_for(w.R)) {
      case 4: k_finish<4><<<fb, 256, 0, s>>>(f); break;
      case 8: k_finish<8><<<fb, 256, 0, s>>>(f); break;
      case 16: k_scale<16><<<fb, 256, 0, s>>>(f); break;
      default: k_scale<32><<<fb, 256, 0, s>>>(f); break;
    }
    ADATM_LAUNCH();
  }
  // BF16 factors were rounded after the Gram was taken: take it again from
  // the rounded rows, so the next modes' normal equations use the factor the
  // MTTKRPs read
  if (Ab) gram(A, rows, w.R, w.ldr, G_mode, w, s, true);
  if (inner && fit_grams != nullptr && !f.fit) fit(*fit_grams, w, s);
}

int update_kernels(uint64_t rows, bool bf16, const AlsWork &w) {
  const int nb = update_blocks(rows, w.R, w.nblocks);
  if (last_finishes(nb, w.R)) return bf16 ? 2 : 1;
  return (one_finish(w.R) ? 2 : 3) + (bf16 ? 2 : 0);
}

void fit(const GramSet &g, AlsWork &w, cudaStream_t s) {
  k_fit<<<1, 256, 0, s>>>(g, w.nmodes, w.R, w.lambda.get(), w.part_inner.get(), w.inner_blocks,
                          w.scalars.get(), w.fit_trace.get(), w.max_trace, w.iter.get());
  ADATM_LAUNCH();
}

// ---------------------------------------------------------------------------
// G = A^T A without any device allocation.
//
// For callers that cannot allocate device memory at the point of the call:
// a host whose caching allocator already holds nearly all of HBM (cudaMalloc
// would fail there), or a loop that must not pay cudaFree's implicit
// device-wide synchronisation. The per-block partial Grams and column maxima
// live in a fixed file-scope device array instead of an AlsWork, which bounds
// the rank to kNoallocMaxR columns and the row blocks to kNoallocBlocks.
//
// Every block of k_update writes its whole partial before k_finalize reads
// it, so nothing in the scratch has to start at zero. The scratch is shared
// by all calls on one device: calls that overlap in time (two host threads,
// or streams not ordered against each other) race on it. The first call on a
// device resolves the scratch address (and sets kernel attributes), which is
// set-up work a caller should do once before any stream capture.
// ---------------------------------------------------------------------------
constexpr int kNoallocMaxR = 64;
constexpr int kNoallocBlocks = 64;
constexpr size_t kNoallocGramDoubles = (size_t)kNoallocBlocks * kNoallocMaxR * kNoallocMaxR;
constexpr size_t kNoallocDoubles = kNoallocGramDoubles + (size_t)kNoallocBlocks * kNoallocMaxR;
constexpr int kNoallocMaxDevices = 64;

// 2 MiB of partial Grams + 32 KiB of column maxima.
static __device__ __align__(256) double g_noalloc_scratch[kNoallocDoubles];

namespace {

struct NoallocSlot {
  std::mutex mu;
  bool ready = false;
  double *ptr = nullptr;
};
NoallocSlot g_noalloc_slots[kNoallocMaxDevices];

// Device address of the scratch on the current device, resolved on the
// first successful call and kept; a failed set-up is not kept, so a later
// call tries again. cudaDeviceReset unloads the module that holds the
// scratch: the kept address is then stale, so a process must not call the
// entry point again after resetting the device.
double *noalloc_scratch() {
  int dev = 0;
  ADATM_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kNoallocMaxDevices) throw BadInput("device ordinal above the scratch table");
  NoallocSlot &slot = g_noalloc_slots[dev];
  std::lock_guard<std::mutex> lk(slot.mu);
  if (!slot.ready) {
    void *p = nullptr;
    const cudaError_t err = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (err != cudaSuccess) {
      cudaGetLastError();
      throw CudaError(std::string("scratch set-up failed: ") + cudaGetErrorString(err));
    }
    set_attributes();
    slot.ptr = static_cast<double *>(p);
    slot.ready = true;
  }
  return slot.ptr;
}

}  // namespace

int gram_noalloc_max_rank() { return kNoallocMaxR; }

void gram_noalloc(const float *A, uint64_t rows, int R, int ldr, double *G, cudaStream_t s) {
  if (R < 1 || R > kNoallocMaxR)
    throw BadInput("adatm_gram_noalloc: R = " + std::to_string(R) + " is outside 1.." +
                   std::to_string(kNoallocMaxR) + ", the columns its fixed scratch holds");
  if (ldr < R || ldr % 4 != 0) throw BadInput("adatm_gram_noalloc: ldr must be >= R and a multiple of 4");
  if (((uintptr_t)A & 15) != 0) throw BadInput("adatm_gram_noalloc: A must be 16-byte aligned");
  double *scratch = noalloc_scratch();
  UpdArgs u = {};
  u.split = 1;
  u.M = A;
  u.rows = rows;
  u.R = R;
  u.ldr = ldr;
  u.part_gram = scratch;
  u.part_max = scratch + kNoallocGramDoubles;
  const int nb = update_blocks(rows, R, kNoallocBlocks);
  run_update(u, nb, s);
  k_finalize<<<finalize_blocks(R), 256, 0, s>>>(finish_args(u, nb, G));
  ADATM_LAUNCH();
}

}  // namespace adatm
