// dlnL/dQ: the plan's dlnL/dP chained through P = exp(Q t r) in the eigenbasis
// of Q = U diag(lambda) W (the Frechet derivative of the matrix exponential):
//
//   M = U^T G W^T,   X = sum_(branch, k) F(t r) .* M,   dlnL/dQ = W^T X U^T,
//   F_mn = (e^(lambda_m tau) - e^(lambda_n tau)) / (lambda_m - lambda_n)
//        = tau e^(max) phi(-|lambda_m - lambda_n| tau),  phi(z) = expm1(z) / z,
//   dlnL/dtau = sum_m lambda_m e^(lambda_m tau) M_mm  (-> branch lengths, rates).
//
// Unlike the chain through dU, dW (tt_pmatrix.cuh, tt_wide.cuh) nothing here
// differentiates eigenvectors, so the result is well conditioned at any
// working precision: FP32 plans of the wide path run these products in FP32.
#include <algorithm>
#include <string>

#include "../../include/torchtree_gb300.h"
#include "tt_plan.h"
#include "tt_wide.cuh"

namespace tt {

namespace {

// F_mn from the states' exponentials em = exp(am),
// en = exp(an) (am = lambda_m tau, an = lambda_n tau), FP32: far apart,
// tau (em - en) / (am - an) has no cancellation; within 0.5, the Taylor
// series of expm1(x) / x to x^7 (remainder below 1.1e-8 for |x| <= 0.5).
__device__ __forceinline__ float frechet_e(float am, float an, float em, float en, float tau) {
  const float d = am - an;
  if (fabsf(d) > 0.5f) return tau * (em - en) / d;
  const float x = -fabsf(d);
  float phi = 1.0f / 40320.0f;
  phi = fmaf(phi, x, 1.0f / 5040.0f);
  phi = fmaf(phi, x, 1.0f / 720.0f);
  phi = fmaf(phi, x, 1.0f / 120.0f);
  phi = fmaf(phi, x, 1.0f / 24.0f);
  phi = fmaf(phi, x, 1.0f / 6.0f);
  phi = fmaf(phi, x, 0.5f);
  phi = fmaf(phi, x, 1.0f);
  return tau * fmaxf(em, en) * phi;
}

// The same in FP64, as tau sqrt(em en) sinh(delta) / delta with delta = (am - an) / 2
// and hm = exp(am / 2), hn likewise: the even Taylor series (all terms positive, so
// no cancellation) to delta^14 for |delta| <= 1/2 and to delta^24 for
// |delta| <= 2 (remainders below 5e-20 and 7e-21); beyond, (em - en) /
// (am - an) has none (1 - e^-4).  About 11 FP64 instructions per pair where exp,
// expm1 and the division took 70 (FP64 instructions are the time here).
__device__ __forceinline__ double frechet_e(double am, double an, double hm, double hn, double tau) {
  const double delta = 0.5 * (am - an), x = delta * delta;
  double s;
  if (x <= 0.25) {
    s = 1.0 / 1307674368000.0;  // 1 / 15!
    s = fma(s, x, 1.0 / 6227020800.0);
    s = fma(s, x, 1.0 / 39916800.0);
    s = fma(s, x, 1.0 / 362880.0);
    s = fma(s, x, 1.0 / 5040.0);
    s = fma(s, x, 1.0 / 120.0);
    s = fma(s, x, 1.0 / 6.0);
    s = fma(s, x, 1.0);
  } else if (x <= 4.0) {
    s = 1.0 / 15511210043330985984000000.0;  // 1 / 25!
    s = fma(s, x, 1.0 / 25852016738884976640000.0);
    s = fma(s, x, 1.0 / 51090942171709440000.0);
    s = fma(s, x, 1.0 / 121645100408832000.0);
    s = fma(s, x, 1.0 / 355687428096000.0);
    s = fma(s, x, 1.0 / 1307674368000.0);
    s = fma(s, x, 1.0 / 6227020800.0);
    s = fma(s, x, 1.0 / 39916800.0);
    s = fma(s, x, 1.0 / 362880.0);
    s = fma(s, x, 1.0 / 5040.0);
    s = fma(s, x, 1.0 / 120.0);
    s = fma(s, x, 1.0 / 6.0);
    s = fma(s, x, 1.0);
  } else {
    return tau * (hm * hm - hn * hn) / (am - an);
  }
  return tau * (hm * hn) * s;
}

// what frechet_e takes of a state: exp(a) in FP32, exp(a / 2) in FP64
__device__ __forceinline__ float frechet_exp(float, float e) { return e; }
__device__ __forceinline__ double frechet_exp(double a, double) { return exp(0.5 * a); }
__device__ __forceinline__ float exp_t(float x) { return expf(x); }
__device__ __forceinline__ double exp_t(double x) { return exp(x); }

}  // namespace

// 4 states, FP32 plans: one CTA per (chunk of 128 branches, sample), one branch
// per thread, products in FP32, sums over a thread's categories in FP32 and
// across the CTA in FP64; X and the rate sums reduced in a fixed order through
// shared memory.  Chunk partials [S*S + K].
__global__ void __launch_bounds__(128) qgrad_small_f32_kernel(const double *G, const double *lam, const double *U,
                                                          const double *W, const double *bl, const double *rates,
                                                          int B, int K, double *part, double *dbl) {
  using T = float;
  constexpr int S = 4;
  __shared__ double red[128][S * S + 8];
  const int chunk = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  T u[S][S], w[S][S], l[S];
#pragma unroll
  for (int i = 0; i < S; ++i) {
    l[i] = T(lam[b * S + i]);
#pragma unroll
    for (int j = 0; j < S; ++j) {
      u[i][j] = T(U[(size_t(b) * S + i) * S + j]);
      w[i][j] = T(W[(size_t(b) * S + i) * S + j]);
    }
  }
  T X[S][S];
  double dr[8];
#pragma unroll
  for (int i = 0; i < S; ++i)
#pragma unroll
    for (int j = 0; j < S; ++j) X[i][j] = T(0);
#pragma unroll
  for (int k = 0; k < 8; ++k) dr[k] = 0.0;
  for (int br = chunk * 128 + tid; br < min(B, chunk * 128 + 128); br += 128) {
    const double t = bl[size_t(b) * B + br];
    double dt = 0.0;
    for (int k = 0; k < K; ++k) {
      const T tau = T(t * rates[b * K + k]);
      const double *g = G + ((size_t(b) * B + br) * K + k) * S * S;
      T h[S][S], M[S][S];
#pragma unroll
      for (int i = 0; i < S; ++i)
#pragma unroll
        for (int n = 0; n < S; ++n) {
          T acc = T(0);
#pragma unroll
          for (int j = 0; j < S; ++j) acc = fma(T(g[i * S + j]), w[n][j], acc);
          h[i][n] = acc;
        }
#pragma unroll
      for (int m = 0; m < S; ++m)
#pragma unroll
        for (int n = 0; n < S; ++n) {
          T acc = T(0);
#pragma unroll
          for (int i = 0; i < S; ++i) acc = fma(u[i][m], h[i][n], acc);
          M[m][n] = acc;
        }
      T sk = T(0);
      {  // the states' exponentials once, the divided differences from them
        T lt[S], es[S];
#pragma unroll
        for (int m = 0; m < S; ++m) {
          lt[m] = l[m] * tau;
          es[m] = exp_t(lt[m]);
        }
#pragma unroll
        for (int m = 0; m < S; ++m) {
          sk = fma(l[m] * es[m], M[m][m], sk);
#pragma unroll
          for (int n = 0; n < S; ++n) X[m][n] = fma(frechet_e(lt[m], lt[n], es[m], es[n], tau), M[m][n], X[m][n]);
        }
      }
      const double s = double(sk);
      dt = fma(s, rates[b * K + k], dt);
      if (k < 8) dr[k] = fma(s, t, dr[k]);
    }
    if (dbl) dbl[size_t(b) * B + br] = dt;
  }
#pragma unroll
  for (int i = 0; i < S; ++i)
#pragma unroll
    for (int j = 0; j < S; ++j) red[tid][i * S + j] = double(X[i][j]);
#pragma unroll
  for (int k = 0; k < 8; ++k) red[tid][S * S + k] = dr[k];
  __syncthreads();
  for (int e = tid; e < S * S + K; e += 128) {
    double acc = 0.0;
    for (int r = 0; r < 128; ++r) acc += red[r][e];
    part[(size_t(b) * gridDim.x + chunk) * (S * S + K) + e] = acc;
  }
}

// 4 states, FP64 plans, whose instructions are the time: one (branch, category)
// per thread, so that the items spread over more SMs.  The CTA's sum in a fixed
// order through shared memory, and each item's sum_m lambda_m e^(lambda_m tau)
// M_mm.  500 tips x 4 samples: 140 us (a branch per thread, exp and expm1 per
// pair) -> 19 us.
__global__ void __launch_bounds__(128) qgrad_small_f64_kernel(const double *G, const double *lam, const double *U,
                                                          const double *W, const double *bl, const double *rates,
                                                          int B, int K, double *part, double *sdiag) {
  using T = double;
  constexpr int S = 4;
  __shared__ double red[128][S * S + 1], seg[8][S * S];
  const int chunk = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
  const int item = chunk * 128 + tid;
  T X[S][S];
#pragma unroll
  for (int i = 0; i < S; ++i)
#pragma unroll
    for (int j = 0; j < S; ++j) X[i][j] = T(0);
  if (item < B * K) {
    const int br = item / K, k = item - br * K;
    T u[S][S], w[S][S], l[S], lt[S], es[S], hx[S], h[S][S];
    const T tau = bl[size_t(b) * B + br] * rates[b * K + k];
    const double *g = G + (size_t(b) * B * K + item) * S * S;
#pragma unroll
    for (int i = 0; i < S; ++i) {
      l[i] = lam[b * S + i];
#pragma unroll
      for (int j = 0; j < S; ++j) {
        u[i][j] = U[(size_t(b) * S + i) * S + j];
        w[i][j] = W[(size_t(b) * S + i) * S + j];
      }
    }
#pragma unroll
    for (int i = 0; i < S; ++i)
#pragma unroll
      for (int n = 0; n < S; ++n) {
        T acc = T(0);
#pragma unroll
        for (int j = 0; j < S; ++j) acc = fma(g[i * S + j], w[n][j], acc);
        h[i][n] = acc;
      }
#pragma unroll
    for (int m = 0; m < S; ++m) {
      lt[m] = l[m] * tau;
      es[m] = exp(lt[m]);
      hx[m] = exp(0.5 * lt[m]);
#pragma unroll
      for (int n = 0; n < S; ++n) {
        T acc = T(0);
#pragma unroll
        for (int i = 0; i < S; ++i) acc = fma(u[i][m], h[i][n], acc);
        X[m][n] = acc;
      }
    }
    T sk = T(0);
#pragma unroll
    for (int m = 0; m < S; ++m) sk = fma(l[m] * es[m], X[m][m], sk);
#pragma unroll
    for (int m = 0; m < S; ++m)
#pragma unroll
      for (int n = m; n < S; ++n) {  // F is symmetric
        const T f = frechet_e(lt[m], lt[n], hx[m], hx[n], tau);
        X[m][n] *= f;
        if (n > m) X[n][m] *= f;
      }
    sdiag[size_t(b) * B * K + item] = sk;
  }
#pragma unroll
  for (int i = 0; i < S; ++i)
#pragma unroll
    for (int j = 0; j < S; ++j) red[tid][i * S + j] = X[i][j];
  __syncthreads();
  {
    const int e = tid & 15, q = tid >> 4;
    double acc = 0.0;
#pragma unroll
    for (int r = 0; r < 16; ++r) acc += red[q * 16 + r][e];
    seg[q][e] = acc;
  }
  __syncthreads();
  if (tid < S * S) {
    double acc = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) acc += seg[q][tid];
    part[(size_t(b) * gridDim.x + chunk) * S * S + tid] = acc;
  }
}

// 20 / 61 states: one CTA per (run of ipc (branch, category) items, sample,
// slab of NS columns); per item H = G W^T and M = U^T H over the slab as 4 x 4
// register tiles (rows ib + IB x, columns n0 + jb + JB y), then X += F .* M in the
// thread's tile.  A run's X goes out in FP64, and per item the slab's part of
// sum_m lambda_m e^(lambda_m tau) M_mm.
//
// Bound by FP64 arithmetic in FP64 plans, so an item is split over two slabs and
// a run is as short as one item: 472 items of one small codon set kept 15 CTAs
// busy before (8 branches each), now 944.  20 states: one warp per CTA (25 of
// 32 lanes hold a tile).  60 taxa, 61 states, FP64, 1 sample: 6,171 (exp and expm1
// per pair of states, 8 branches per CTA) -> 520 us.
//
// FP32 plans of 20 states are bound by an item's chain of dependent phases: the
// products unrolled over all 20 states, only the diagonal tiles' threads in the
// diagonal sum (in FP64, 64 cycles an addition), and three further warps that stage
// G and add that sum up while the first goes on.  30 taxa x 4 categories 189 (one warp,
// the sum by shuffles over all lanes) -> 152 us, the three launches together.
template <typename T, int SP, int NS>
struct QgradCfg {
  static constexpr int IB = SP / 4, JB = NS / 4, TILES = IB * JB;
  static constexpr bool kChain = sizeof(T) == 4 && SP == 20;
  static constexpr int NT = kChain ? 128 : (TILES + 31) / 32 * 32;
  static constexpr int GS = SP + 4;  // row stride of the transposed G (its stores are down a column)
  static constexpr int SLABS = SP / NS;
  static constexpr int SUMS = kChain ? IB : NT / 32;  // parts of the diagonal sum
  static constexpr size_t smem() {
    return sizeof(T) * (SP * SP + 2 * SP * NS + SP * GS + 4 * SP) + sizeof(double) * SUMS;
  }
};

template <typename T, int SP, int NS>
__global__ void __launch_bounds__(QgradCfg<T, SP, NS>::NT)
    wide_qgrad_kernel(const double *G, const double *lam, const double *U, const double *W, const double *bl,
                      const double *rates, int S, int B, int K, int ipc, double *sdiag, double *part) {
  using C = QgradCfg<T, SP, NS>;
  constexpr int IB = C::IB, JB = C::JB, NT = C::NT, GS = C::GS;
  extern __shared__ __align__(128) unsigned char smem[];
  T *ug = reinterpret_cast<T *>(smem);  // [i][perm m] = U[i][m]
  T *wt = ug + SP * SP;                  // [j][perm n] = W[n0 + n][j]
  T *hs = wt + SP * NS;                  // [i][perm n] = H[i][n0 + n]
  T *gt = hs + SP * NS;                  // [j][perm i] = G[i][j], rows GS apart
  T *ls = gt + SP * GS;                  // lambda [SP]
  T *lt = ls + SP;                       // lambda tau [SP]
  T *es = lt + SP;                       // exp(lambda tau) [SP]
  T *hx = es + SP;                       // frechet_exp [SP]
  double *dred = reinterpret_cast<double *>(hx + SP);  // [SUMS] parts of the diagonal sum
  const int chunk = blockIdx.x, b = blockIdx.y, n0 = blockIdx.z * NS, tid = threadIdx.x;
  const int items = B * K, i0 = chunk * ipc, i1 = min(items, i0 + ipc);
  const bool tile = tid < C::TILES;
  const int bm = tile ? tid / JB : 0, bn = tile ? tid - bm * JB : 0;
  for (int e = tid; e < SP * SP; e += NT) {
    const int x = e / SP, y = e - x * SP;
    ug[x * SP + wperm<IB>(y)] = (x < S && y < S) ? T(U[(size_t(b) * S + x) * S + y]) : T(0);
  }
  for (int e = tid; e < SP * NS; e += NT) {
    const int n = e / SP, j = e - n * SP;
    wt[j * NS + wperm<JB>(n)] = (n0 + n < S && j < S) ? T(W[(size_t(b) * S + n0 + n) * S + j]) : T(0);
  }
  for (int m = tid; m < SP; m += NT) ls[m] = m < S ? T(lam[size_t(b) * S + m]) : T(0);
  T X[4][4];
#pragma unroll
  for (int x = 0; x < 4; ++x)
#pragma unroll
    for (int y = 0; y < 4; ++y) X[x][y] = T(0);
  // one-warp CTAs: the next item's G travels in registers while this one computes
  constexpr bool kAhead = NT == 32;
  constexpr int GR = kAhead ? (SP * SP + NT - 1) / NT : 1;
  double ahead[GR];
  auto fetch = [&](int item) {
    const double *g = G + (size_t(b) * items + item) * S * S;
#pragma unroll
    for (int r = 0; r < GR; ++r) {
      const int e = tid + r * NT, i = e / SP, j = e - i * SP;
      ahead[r] = (i < S && j < S) ? g[i * S + j] : 0.0;
    }
  };
  if (kAhead) fetch(i0);
  for (int item = i0; item < i1; ++item) {
    const int br = item / K, k = item - br * K;
    const T tau = T(bl[size_t(b) * B + br] * rates[size_t(b) * K + k]);
    __syncthreads();  // the previous item is done with gt / hs / es (and ls is there)
    for (int m = tid; m < SP; m += NT) {
      lt[m] = ls[m] * tau;
      const T ex = exp_t(ls[m] * tau);
      es[m] = m < S ? ex : T(0);
      hx[m] = m < S ? frechet_exp(ls[m] * tau, ex) : T(0);
    }
    if constexpr (kAhead) {
#pragma unroll
      for (int r = 0; r < GR; ++r) {
        const int e = tid + r * NT, i = e / SP, j = e - i * SP;
        if (i < SP) gt[j * GS + wperm<IB>(i)] = T(ahead[r]);
      }
      if (item + 1 < i1) fetch(item + 1);
    } else {
      const double *g = G + (size_t(b) * items + item) * S * S;
      for (int e = tid; e < SP * SP; e += NT) {
        const int i = e / SP, j = e - i * SP;
        gt[j * GS + wperm<IB>(i)] = (i < S && j < S) ? T(g[i * S + j]) : T(0);
      }
    }
    __syncthreads();
    if (tile) {  // H block: rows i = bm + IB x, columns n = n0 + bn + JB y
      T h[4][4];
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) h[x][y] = T(0);
      auto step = [&](int j) {
        T ga[4], wa[4];
        V4<T>::ld(gt + j * GS + bm * 4, ga);
        V4<T>::ld(wt + j * NS + bn * 4, wa);
        outer4(h, ga, wa);
      };
      if constexpr (C::kChain) {
#pragma unroll
        for (int j = 0; j < SP; ++j) step(j);
      } else {
#pragma unroll 4
        for (int j = 0; j < S; ++j) step(j);
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) V4<T>::st(hs + (bm + IB * x) * NS + bn * 4, h[x]);
    }
    __syncthreads();
    double dsum = 0.0;
    if (tile) {  // M block: rows m = bm + IB x, columns n = n0 + bn + JB y
      T M[4][4];
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) M[x][y] = T(0);
      auto step = [&](int i) {
        T ua[4], ha[4];
        V4<T>::ld(ug + i * SP + bm * 4, ua);
        V4<T>::ld(hs + i * NS + bn * 4, ha);
        outer4(M, ua, ha);
      };
      if constexpr (C::kChain) {
#pragma unroll
        for (int i = 0; i < SP; ++i) step(i);
      } else {
#pragma unroll 4
        for (int i = 0; i < S; ++i) step(i);
      }
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const int m = bm + IB * x;
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          const int n = n0 + bn + JB * y;
          X[x][y] += frechet_e(lt[m], lt[n], hx[m], hx[n], tau) * M[x][y];
          if (!C::kChain && m == n && m < S) dsum += double(ls[m] * es[m] * M[x][y]);
        }
      }
      if (C::kChain && bm == bn) {  // (one slab, square: the diagonal lies in these tiles)
#pragma unroll
        for (int x = 0; x < 4; ++x) {
          const int m = bm + IB * x;
          if (m < S) dsum += double(ls[m] * es[m] * M[x][x]);
        }
        dred[bm] = dsum;
      }
    }
    if constexpr (!C::kChain) {
      dsum = warp_sum(dsum);
      if ((tid & 31) == 0) dred[tid >> 5] = dsum;
    }
    __syncthreads();
    if (tid == (C::kChain ? NT - 1 : 0)) {  // fixed order
      double s = 0.0;
#pragma unroll
      for (int w = 0; w < C::SUMS; ++w) s += dred[w];
      sdiag[(size_t(blockIdx.z) * gridDim.y + b) * items + item] = s;
    }
  }
  double *dst = part + (size_t(b) * gridDim.x + chunk) * S * S;
  if (tile)
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const int m = bm + IB * x, n = n0 + bn + JB * y;
        if (m < S && n < S) dst[m * S + n] = double(X[x][y]);
      }
}

// per sample, kQRows rows per CTA (grid: row blocks x samples), FP64:
// X rows = sums of the runs' partials, then Z rows = X rows U^T; spreading the
// rows over CTAs keeps the FP64 work off a single SM per sample.  The CTAs also
// share the branch lengths' gradients dt = sum_k s r_k (s: the item's diagonal
// sum over its slabs), the first sums the rates' dr_k = sum_branches s t; without
// item sums (sdiag NULL) the lengths are written and the partials hold the rates.
constexpr int kQRows = 4;

__global__ void __launch_bounds__(256) qgrad_sum_rows_kernel(const double *part, int nchunks, int width, const double *sdiag,
                                                             int slabs, const double *U, const double *bl,
                                                             const double *rates, int S, int B, int K, double *Z,
                                                             double *dbl, double *drates) {
  __shared__ double X[kQRows][64];
  const int b = blockIdx.y, r0 = blockIdx.x * kQRows, tid = threadIdx.x;
  const int rows = min(kQRows, S - r0);
  for (int e = tid; e < rows * S; e += blockDim.x) {
    const int r = e / S, c = e - r * S;
    const double *src = part + size_t(b) * nchunks * width + (r0 + r) * S + c;
    double s = 0.0;
#pragma unroll 8
    for (int ch = 0; ch < nchunks; ++ch) s += src[size_t(ch) * width];
    X[r][c] = s;
  }
  if (!sdiag && blockIdx.x == 0 && drates)  // the partials hold the rates' sums
    for (int k = tid; k < K; k += blockDim.x) {
      double s = 0.0;
      for (int ch = 0; ch < nchunks; ++ch) s += part[(size_t(b) * nchunks + ch) * width + S * S + k];
      drates[size_t(b) * K + k] = s;
    }
  auto diag = [&](int br, int k) {
    double s = 0.0;
    for (int z = 0; z < slabs; ++z) s += sdiag[(size_t(z) * gridDim.y + b) * B * K + size_t(br) * K + k];
    return s;
  };
  if (sdiag && dbl)
    for (int br = blockIdx.x * 256 + tid; br < B; br += gridDim.x * 256) {
      double dt = 0.0;
      for (int k = 0; k < K; ++k) dt = fma(diag(br, k), rates[size_t(b) * K + k], dt);
      dbl[size_t(b) * B + br] = dt;
    }
  if (sdiag && blockIdx.x == 0 && drates)
    for (int k = tid >> 5; k < K; k += 8) {
      double dr = 0.0;
      for (int br = tid & 31; br < B; br += 32) dr = fma(diag(br, k), bl[size_t(b) * B + br], dr);
      dr = warp_sum(dr);
      if ((tid & 31) == 0) drates[size_t(b) * K + k] = dr;
    }
  __syncthreads();
  const double *u = U + size_t(b) * S * S;
  for (int e = tid; e < rows * S; e += blockDim.x) {  // Z[m][j] = sum_n X[m][n] U[j][n]
    const int r = e / S, j = e - r * S;
    double acc = 0.0;
    for (int n = 0; n < S; ++n) acc = fma(X[r][n], u[j * S + n], acc);
    Z[(size_t(b) * S + r0 + r) * S + j] = acc;
  }
}

// dQ rows i = sum_m W[m][i] Z[m][j], kQRows rows per CTA, FP64.
__global__ void __launch_bounds__(256) qgrad_dq_rows_kernel(const double *Z, const double *W, int S, double *dQ) {
  const int b = blockIdx.y, r0 = blockIdx.x * kQRows, tid = threadIdx.x;
  const int rows = min(kQRows, S - r0);
  const double *w = W + size_t(b) * S * S, *z = Z + size_t(b) * S * S;
  for (int e = tid; e < rows * S; e += blockDim.x) {
    const int i = r0 + e / S, j = e - (e / S) * S;
    double acc = 0.0;
    for (int m = 0; m < S; ++m) acc = fma(w[m * S + i], z[m * S + j], acc);
    dQ[size_t(b) * S * S + size_t(i) * S + j] = acc;
  }
}

namespace {

// (branch, category) items per CTA, CTAs per sample and slabs of an item's
// columns.  FP32 plans: eight branches per CTA (their sum is in FP32, so its
// length is a matter of precision).  FP64: runs of one item until the CTAs make
// four waves of those resident per SM (two in codon plans, 16 one-warp CTAs at 20
// states), then longer runs (fewer partial sums).
struct QgradPlan {
  int ipc, nchunks, slabs, width;
};

QgradPlan qgrad_plan(const tt_plan *p) {
  const long long items = (long long)p->B * p->K;
  const bool f64 = p->precision == TT_PRECISION_F64, narrow = p->S <= 20;
  QgradPlan q{f64 ? 128 : 128 * p->K, 0, 1, p->S * p->S};
  if (p->S == 4 && !f64) q.width += p->K;
  if (p->S != 4) {
    q.slabs = narrow || !f64 ? 1 : 2;
    q.ipc = f64 ? int(std::max(1ll, items * p->batch * q.slabs / (4ll * 152 * (narrow ? 16 : 2)))) : 8 * p->K;
  }
  q.nchunks = int((items + q.ipc - 1) / q.ipc);
  return q;
}

template <typename T, int SP, int NS>
cudaError_t launch_wide_qgrad(tt_plan *p, const double *lam, const double *U, const double *W, const double *bl,
                              const double *rates, double *sdiag, double *part, const QgradPlan &q, cudaStream_t s) {
  using C = QgradCfg<T, SP, NS>;
  constexpr size_t smem = C::smem();
  cudaError_t e = kernel_smem(wide_qgrad_kernel<T, SP, NS>, smem, true);
  if (e != cudaSuccess) return e;
  wide_qgrad_kernel<T, SP, NS><<<dim3(q.nchunks, p->batch, C::SLABS), C::NT, smem, s>>>(
      p->d_G, lam, U, W, bl, rates, p->S, p->B, p->K, q.ipc, sdiag, part);
  return cudaGetLastError();
}

}  // namespace

int rate_matrix_gradient(tt_plan *p, const double *lam, const double *U, const double *W, const double *bl,
                         const double *rates, double *dQ, double *dbl, double *drates, cudaStream_t s) {
  const int S = p->S, K = p->K;
  const QgradPlan q = qgrad_plan(p);
  const size_t n_part = size_t(p->batch) * q.nchunks * q.width, n_z = size_t(p->batch) * S * S;
  const size_t n_diag = size_t(q.slabs) * p->batch * p->B * K;
  cudaError_t e = cudaSuccess;
  if (!p->d_qpart) {  // allocated on first use: the runs' partials, Z [b][S][S] of the finishing step, diagonal sums
    e = cudaMalloc(reinterpret_cast<void **>(&p->d_qpart), (n_part + n_z + n_diag) * sizeof(double));
    if (e != cudaSuccess) {
      cudaGetLastError();
      return record_error(TT_ERR_OUT_OF_MEMORY, "cudaMalloc of the rate-matrix gradient chunks failed");
    }
    p->bytes += (n_part + n_z + n_diag) * sizeof(double);
  }
  double *part = p->d_qpart, *Z = part + n_part, *sdiag = Z + n_z;
  const bool f32 = p->precision == TT_PRECISION_F32;
  if (S == 4) {
    const dim3 grid(q.nchunks, p->batch);
    if (f32)
      qgrad_small_f32_kernel<<<grid, 128, 0, s>>>(p->d_G, lam, U, W, bl, rates, p->B, K, part, dbl);
    else
      qgrad_small_f64_kernel<<<grid, 128, 0, s>>>(p->d_G, lam, U, W, bl, rates, p->B, K, part, sdiag);
    e = cudaGetLastError();
  } else if (S <= 20) {
    e = f32 ? launch_wide_qgrad<float, 20, 20>(p, lam, U, W, bl, rates, sdiag, part, q, s)
            : launch_wide_qgrad<double, 20, 20>(p, lam, U, W, bl, rates, sdiag, part, q, s);
  } else {
    e = f32 ? launch_wide_qgrad<float, 64, 64>(p, lam, U, W, bl, rates, sdiag, part, q, s)
            : launch_wide_qgrad<double, 64, 32>(p, lam, U, W, bl, rates, sdiag, part, q, s);
  }
  if (e == cudaSuccess) {
    const dim3 grid((S + kQRows - 1) / kQRows, p->batch);
    qgrad_sum_rows_kernel<<<grid, 256, 0, s>>>(part, q.nchunks, q.width, S == 4 && f32 ? nullptr : sdiag, q.slabs, U, bl, rates, S, p->B, K, Z, dbl,
                                               drates);
    if (dQ) qgrad_dq_rows_kernel<<<grid, 256, 0, s>>>(Z, W, S, dQ);
    e = cudaGetLastError();
  }
  p->launches += dQ ? 3 : 2;
  if (e != cudaSuccess)
    return record_error(e == cudaErrorMemoryAllocation ? TT_ERR_OUT_OF_MEMORY : TT_ERR_CUDA,
                        (std::string("rate-matrix gradient launch: ") + cudaGetErrorString(e)).c_str());
  return TT_OK;
}

}  // namespace tt
