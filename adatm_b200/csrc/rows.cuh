// rows.cuh -- rows of R columns spread over the lanes of a warp: loads of FP32
// and BF16 factor rows, packed FP32 products.
#pragma once

#include "pull.cuh"

namespace adatm {

template <int V>
struct alignas(sizeof(float) * V) fv {
  float x[V];
};

// Pairs of columns go through the packed FP32 instructions (one issue slot
// for two products; each is rounded as its scalar form is).
__device__ __forceinline__ uint64_t pack2(float x, float y) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t p, float &x, float &y) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(p));
}
// Columns col .. col+3 of factor row `row` (FP32 or BF16 storage).
template <FactorType FT>
__device__ __forceinline__ float4 ld_factor4(const void *U, uint32_t row, int ldr, int col, bool act) {
  if (!act) return make_float4(0.f, 0.f, 0.f, 0.f);
  if constexpr (FT == FactorType::F32) {
    return __ldg(reinterpret_cast<const float4 *>(static_cast<const float *>(U) + (size_t)row * ldr + col));
  } else {
    const uint2 raw = __ldg(
        reinterpret_cast<const uint2 *>(static_cast<const __nv_bfloat16 *>(U) + (size_t)row * ldr + col));
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&raw.x));
    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&raw.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
  }
}

// And of an FP32 row matrix (memo rows).
__device__ __forceinline__ float4 ld_rows4(const float *base, uint64_t row, int ldr, int col, bool act) {
  if (!act) return make_float4(0.f, 0.f, 0.f, 0.f);
  return __ldg(reinterpret_cast<const float4 *>(base + row * (uint64_t)ldr + col));
}

// FP64 output rows: the MTTKRP sums of a row can come from millions of
// units (a skewed slice), and FP32 sums of that many partials lose several
// digits; outputs are stored and added in FP64.
template <int V>
__device__ __forceinline__ void st_out(double *base, uint64_t row, int ldr, int col, const fv<V> &v,
                                       bool act) {
  if (!act) return;
  double *p = base + row * (uint64_t)ldr + col;
  if constexpr (V == 1) {
    *p = v.x[0];
  } else if constexpr (V == 2) {
    *reinterpret_cast<double2 *>(p) = make_double2(v.x[0], v.x[1]);
  } else {
    *reinterpret_cast<double2 *>(p) = make_double2(v.x[0], v.x[1]);
    *reinterpret_cast<double2 *>(p + 2) = make_double2(v.x[2], v.x[3]);
  }
}

// V columns as packed pairs (one register pair for two FP32 columns), the
// form the contraction keeps its rows in: no moves between loads and the
// packed products.
template <int V>
struct alignas(4 * V) Row {
  uint64_t w[V / 2];
};
template <>
struct alignas(4) Row<1> {
  float w;
};
template <int V>
__device__ __forceinline__ Row<V> row_zero() {
  Row<V> r;
  if constexpr (V == 1) {
    r.w = 0.f;
  } else {
#pragma unroll
    for (int i = 0; i < V / 2; ++i) r.w[i] = 0ull;
  }
  return r;
}
template <int V>
__device__ __forceinline__ fv<V> row_values(const Row<V> &r) {
  fv<V> f;
  if constexpr (V == 1) {
    f.x[0] = r.w;
  } else {
#pragma unroll
    for (int i = 0; i < V / 2; ++i) unpack2(r.w[i], f.x[2 * i], f.x[2 * i + 1]);
  }
  return f;
}
template <int V>
__device__ __forceinline__ Row<V> row_mul(const Row<V> &a, const Row<V> &b) {
  Row<V> r;
  if constexpr (V == 1) {
    r.w = a.w * b.w;
  } else {
#pragma unroll
    for (int i = 0; i < V / 2; ++i)
      asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.w[i]) : "l"(a.w[i]), "l"(b.w[i]));
  }
  return r;
}
template <int V>
__device__ __forceinline__ Row<V> row_add(const Row<V> &a, const Row<V> &b) {
  Row<V> r;
  if constexpr (V == 1) {
    r.w = a.w + b.w;
  } else {
#pragma unroll
    for (int i = 0; i < V / 2; ++i)
      asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.w[i]) : "l"(a.w[i]), "l"(b.w[i]));
  }
  return r;
}
template <int V>
__device__ __forceinline__ void row_fma(Row<V> &acc, const Row<V> &a, const Row<V> &b) {
  if constexpr (V == 1) {
    acc.w = fmaf(a.w, b.w, acc.w);
  } else {
#pragma unroll
    for (int i = 0; i < V / 2; ++i)
      asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc.w[i]) : "l"(a.w[i]), "l"(b.w[i]));
  }
}
// A factor row as it is loaded: FP32 columns, or BF16 pairs.
template <int V, FactorType FT>
struct RawRow {
  Row<V> r;
};
template <int V>
struct RawRow<V, FactorType::BF16> {
  uint32_t w[(V + 1) / 2];
};
template <int V, FactorType FT>
__device__ __forceinline__ Row<V> raw_row(const RawRow<V, FT> &a) {
  if constexpr (FT == FactorType::F32) {
    return a.r;
  } else {
    // a BF16 value is the upper half of its FP32 value
    Row<V> r;
    if constexpr (V == 1) {
      r.w = __uint_as_float(a.w[0] << 16);
    } else {
#pragma unroll
      for (int i = 0; i < V / 2; ++i)
        r.w[i] = pack2(__uint_as_float(a.w[i] << 16), __uint_as_float(a.w[i] & 0xFFFF0000u));
    }
    return r;
  }
}
template <int V, FactorType FT>
__device__ __forceinline__ void raw_zero(RawRow<V, FT> &a) {
  if constexpr (FT == FactorType::F32) {
    a.r = row_zero<V>();
  } else {
#pragma unroll
    for (int i = 0; i < (V + 1) / 2; ++i) a.w[i] = 0u;
  }
}
template <int V, FactorType FT>
__device__ __forceinline__ void ld_row(RawRow<V, FT> &a, const char *p) {
  if constexpr (FT == FactorType::F32) {
    if constexpr (V == 1)
      asm("ld.global.nc.f32 %0, [%1];" : "=f"(a.r.w) : "l"(p));
    else if constexpr (V == 2)
      asm("ld.global.nc.b64 %0, [%1];" : "=l"(a.r.w[0]) : "l"(p));
    else
      asm("ld.global.nc.v2.b64 {%0, %1}, [%2];" : "=l"(a.r.w[0]), "=l"(a.r.w[1]) : "l"(p));
  } else {
    if constexpr (V == 1)
      a.w[0] = __ldg(reinterpret_cast<const unsigned short *>(p));
    else if constexpr (V == 2)
      asm("ld.global.nc.b32 %0, [%1];" : "=r"(a.w[0]) : "l"(p));
    else
      asm("ld.global.nc.v2.b32 {%0, %1}, [%2];" : "=r"(a.w[0]), "=r"(a.w[1]) : "l"(p));
  }
}
template <int V, FactorType FT>
__device__ __forceinline__ Row<V> ld_row(const char *p) {
  RawRow<V, FT> a;
  ld_row<V, FT>(a, p);
  return raw_row<V, FT>(a);
}
__device__ __forceinline__ const char *row_at(const char *base, uint32_t row, uint32_t stride) {
  return base + (uint64_t)row * stride;
}
// The tree's arrays are read once, in order: a miss brings the next units
// into L2 as well.
__device__ __forceinline__ uint32_t ld_stream(const uint32_t *p) {
  uint32_t v;
  asm("ld.global.nc.L2::256B.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ float ld_stream(const float *p) {
  float v;
  asm("ld.global.nc.L2::256B.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}
__device__ __forceinline__ uint32_t ld_stream(const uint8_t *p) {
  uint32_t v;
  asm("ld.global.nc.L2::256B.u8 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

// An FP32 row that is read once: it takes no room in L1.
__device__ __forceinline__ void ld_row_once(RawRow<4, FactorType::F32> &a, const char *p) {
  asm("ld.global.nc.L1::no_allocate.v2.b64 {%0, %1}, [%2];" : "=l"(a.r.w[0]), "=l"(a.r.w[1]) : "l"(p));
}

}  // namespace adatm
