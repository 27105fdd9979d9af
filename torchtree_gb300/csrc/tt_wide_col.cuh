// Wide-state post-order of plans with at most 20 states (SP = 20): whole state
// vectors per thread.
//
// Shared memory returns 128 bytes a cycle to an SM's registers, broadcasts
// included, so the words loaded per FMA are what bounds a product of this size.
// The 4 x 4 register tiles of wide_forward_kernel load a word per two FMAs
// (measured: 76 % of the shared-memory bandwidth, half of all stalls), and stage
// both children and the column maximum through shared memory.  Here a thread owns
// kColPatterns<T> patterns and all 20 states: the child's vectors come straight from
// global memory, a matrix row (five 16-byte loads) serves all its patterns, and
// maximum, rescaling and products need no other thread.
//
// A tip child's product is a row of a table formed once per CTA: P times each
// code's vector, with the terms in the order of the matrix product, so its bits
// are the product's (an unambiguous state's row is the matrix's column).  Plans
// with more than kColCodes codes form the product per pattern instead.  Root nodes, and
// in FP32 levels that do not fill the GPU, stay with wide_forward_kernel.  FP32 results do not change by a bit.
//
// 200 taxa x 4,246 patterns x 4 samples, 20 states, FP32: 1,431 -> 789 us (1,112 with
// one pattern per thread).
#pragma once

#include "tt_wide.cuh"

namespace tt {

constexpr int kColStates = 20;
constexpr int kColThreads = 128;
// patterns per thread (consecutive; the registers hold both products in FP32 pairs)
template <typename T>
constexpr int kColPatterns = sizeof(T) == 4 ? 2 : 1;
constexpr int kColCodes = 64;   // tip codes with a product table

// One pattern's 20 values; FP32 as pairs of rows for packed FMAs.
template <typename T>
struct ColVec;
template <>
struct ColVec<float> {
  float2 v[10];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 10; ++i) v[i] = make_float2(0.0f, 0.0f);
  }
  __device__ __forceinline__ void fma_row(const float *row, float x) {  // += row * x
    const float2 xx = make_float2(x, x);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const float4 r = reinterpret_cast<const float4 *>(row)[q];
      v[2 * q] = __ffma2_rn(make_float2(r.x, r.y), xx, v[2 * q]);
      v[2 * q + 1] = __ffma2_rn(make_float2(r.z, r.w), xx, v[2 * q + 1]);
    }
  }
  __device__ __forceinline__ void load(const float *row) {
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const float4 r = reinterpret_cast<const float4 *>(row)[q];
      v[2 * q] = make_float2(r.x, r.y);
      v[2 * q + 1] = make_float2(r.z, r.w);
    }
  }
  __device__ __forceinline__ float get(int i) const { return i & 1 ? v[i >> 1].y : v[i >> 1].x; }
  __device__ __forceinline__ void set(int i, float x) {
    if (i & 1) v[i >> 1].y = x;
    else v[i >> 1].x = x;
  }
};
template <>
struct ColVec<double> {
  double v[20];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 20; ++i) v[i] = 0.0;
  }
  __device__ __forceinline__ void fma_row(const double *row, double x) {
#pragma unroll
    for (int q = 0; q < 10; ++q) {
      const double2 r = reinterpret_cast<const double2 *>(row)[q];
      v[2 * q] = fma(r.x, x, v[2 * q]);
      v[2 * q + 1] = fma(r.y, x, v[2 * q + 1]);
    }
  }
  __device__ __forceinline__ void load(const double *row) {
#pragma unroll
    for (int q = 0; q < 10; ++q) {
      const double2 r = reinterpret_cast<const double2 *>(row)[q];
      v[2 * q] = r.x;
      v[2 * q + 1] = r.y;
    }
  }
  __device__ __forceinline__ double get(int i) const { return v[i]; }
  __device__ __forceinline__ void set(int i, double x) { v[i] = x; }
};

// rescale by the power of two of the largest value; returns its exponent
template <typename T>
__device__ __forceinline__ int col_rescale(ColVec<T> &c) {
  using M = MaxBits<T>;
  typename M::type m = M::zero();
#pragma unroll
  for (int i = 0; i < kColStates; ++i) m = M::larger(m, M::of(c.get(i)));
  const int e = scale_exponent(M::value(m));
#pragma unroll
  for (int i = 0; i < kColStates; ++i) c.set(i, times_pow2_neg(c.get(i), e));
  return e;
}

// tip codes that get a product table
__host__ __device__ inline int col_codes(int C) { return C <= kColCodes ? C : 0; }

template <typename T>
__host__ __device__ inline size_t col_fwd_smem(int C) {
  return sizeof(T) * size_t(2 * kColStates * kColStates + 2 * col_codes(C) * kColStates);
}
// tb[code][i] = sum_j P[i][j] table[code][j] (P row-major), j in order
template <typename T>
__device__ __forceinline__ void col_tip_table(T *tb, const T *P, const T *table, int codes, int tid, int nt) {
  for (int e = tid; e < codes * kColStates; e += nt) {
    const int c = e / kColStates, i = e - c * kColStates;
    T acc = T(0);
#pragma unroll 4
    for (int j = 0; j < kColStates; ++j) acc = fma(P[i * kColStates + j], table[c * kColStates + j], acc);
    tb[e] = acc;
  }
}

// the PP consecutive values of a row at p
template <int PP, typename T>
__device__ __forceinline__ void col_load(T (&x)[PP], const T *p) {
  if constexpr (PP == 2) {
    const float2 f = __ldg(reinterpret_cast<const float2 *>(p));
    x[0] = f.x, x[1] = f.y;
  } else {
    x[0] = __ldg(p);
  }
}

// post-order of internal, non-root nodes: one CTA per (node, run of tiles, sample, category)
template <typename T>
__global__ void __launch_bounds__(kColThreads, 3) wide_col_forward_kernel(const WideArgs<T> a, int code_count) {
  constexpr int SP = kColStates, PP = kColPatterns<T>;
  extern __shared__ __align__(128) unsigned char smem[];
  T *pt = reinterpret_cast<T *>(smem);  // [2][j][i], a tip's as [i][j]
  T *tb = pt + 2 * SP * SP;             // [2][codes][SP]
  const int tid = threadIdx.x, codes = col_codes(code_count);
  const int v = a.nodes[blockIdx.y];
  const int b = blockIdx.z / a.K, k = blockIdx.z - (blockIdx.z / a.K) * a.K;
  const int l = a.left[v - a.tips], r = a.right[v - a.tips];
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int kid = c ? r : l;
    const T *src = a.pmat + ((size_t(b) * a.B + kid) * a.K + k) * SP * SP;
    const bool tab = kid < a.tips && codes > 0;
    for (int ij = tid; ij < SP * SP; ij += kColThreads)
      pt[c * SP * SP + (tab ? ij : (ij % SP) * SP + ij / SP)] = src[ij];
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 2; ++c)
    if ((c ? r : l) < a.tips && codes > 0)
      col_tip_table(tb + c * codes * SP, pt + c * SP * SP, a.table, codes, tid, kColThreads);
  __syncthreads();
  const int t0 = blockIdx.x * a.tiles_per_chunk, t1 = min(a.ntiles, t0 + a.tiles_per_chunk);
  const size_t npad = size_t(a.Npad);
  for (int tile = t0; tile < t1; ++tile) {
    const int n = (tile * kColThreads + tid) * PP;
    if (n >= a.Npad) break;  // Npad is a multiple of 128 and of PP
    ColVec<T> prod[PP];
    int E[PP] = {};
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int kid = c ? r : l;
      ColVec<T> y[PP];
      if (kid < a.tips) {
        const uint8_t *cd = a.codes + size_t(kid) * a.code_stride + n;
#pragma unroll
        for (int q = 0; q < PP; ++q) {
          const int code = cd[q];
          if (code < codes) {
            y[q].load(tb + (c * codes + code) * SP);
          } else if (codes > 0) {  // more codes than when this pass was captured
#pragma unroll
            for (int i = 0; i < SP; ++i) {
              T acc = T(0);
#pragma unroll 1
              for (int j = 0; j < SP; ++j) acc = fma(pt[c * SP * SP + i * SP + j], a.table[code * SP + j], acc);
              y[q].set(i, acc);
            }
          } else {
            y[q].zero();
            for (int j = 0; j < SP; ++j) y[q].fma_row(pt + c * SP * SP + j * SP, a.table[code * SP + j]);
          }
        }
      } else {
        const size_t blk = (size_t(b) * a.I + (kid - a.tips)) * a.K + k;
        const T *src = a.part + blk * SP * npad + n;
        T x[SP][PP];
#pragma unroll
        for (int j = 0; j < SP; ++j) col_load<PP>(x[j], src + j * npad);
#pragma unroll
        for (int q = 0; q < PP; ++q) {
          E[q] += a.expo[blk * npad + n + q];
          y[q].zero();
        }
#pragma unroll
        for (int j = 0; j < SP; ++j)
#pragma unroll
          for (int q = 0; q < PP; ++q) y[q].fma_row(pt + c * SP * SP + j * SP, x[j][q]);
        if (kChildProducts<T> && a.prod) {
          T *pd = a.prod + blk * SP * npad + n;
#pragma unroll
          for (int i = 0; i < SP; ++i)
#pragma unroll
            for (int q = 0; q < PP; ++q) pd[i * npad + q] = y[q].get(i);
        }
      }
#pragma unroll
      for (int q = 0; q < PP; ++q)
#pragma unroll
        for (int i = 0; i < SP; ++i) prod[q].set(i, c == 0 ? y[q].get(i) : prod[q].get(i) * y[q].get(i));
    }
    const size_t blk = (size_t(b) * a.I + (v - a.tips)) * a.K + k;
#pragma unroll
    for (int q = 0; q < PP; ++q) {
      if (a.rescale) E[q] += col_rescale(prod[q]);
      a.expo[blk * npad + n + q] = E[q];
    }
    T *dst = a.part + blk * SP * npad + n;
#pragma unroll
    for (int i = 0; i < SP; ++i) {
      if constexpr (PP == 2)
        *reinterpret_cast<float2 *>(dst + i * npad) = make_float2(prod[0].get(i), prod[1].get(i));
      else
        dst[i * npad] = prod[0].get(i);
    }
  }
}

}  // namespace tt
