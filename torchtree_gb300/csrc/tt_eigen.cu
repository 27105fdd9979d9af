// Per-step model set-up on the device: the eigen system of a reversible rate
// matrix and the discretised Gamma rates, both in FP64.
//
// tt_reversible_eigen replaces the eigendecomposition in
// SymmetricSubstitutionModel.p_t (torchtree/evolution/substitution_model/
// abstract.py:57-79): with Pi = diag(pi), the symmetric matrix
// A = Pi^1/2 Q Pi^-1/2 is diagonalised as A = V diag(lambda) V^T (torch's
// eigh reads the lower triangle; so does this kernel), and
// Q = U diag(lambda) W with U = Pi^-1/2 V, W = V^T Pi^1/2 (V is orthogonal,
// so W is the inverse of U without a matrix inverse).
//
// FP64 arithmetic is scarce on this GPU (a few FP64 FMAs per cycle per SM),
// so the solver does most of its sweeps in FP32 and spreads the FP64 matrix
// products over many CTAs:
//  1. eigen_start_kernel, one or four CTAs per matrix: cyclic Jacobi in FP32 (parallel
//     round-robin ordering of Brent and Luk, 1985; each rotation Golub & Van
//     Loan, Algorithm 8.4.2 "sym.schur2"): eigenvectors X0 good to ~1e-5;
//  2. two Newton-Schulz steps X <- X (3I - X^T X) / 2 (Higham, "Functions of
//     Matrices", 8.3) in FP64, each squaring X's distance from orthonormal
//     (eigen_gram_kernel forms R = I - X^T X, eigen_orth_kernel X <- X + X R/2),
//     kEigRows rows of the products per CTA;
//  3. eigen_gram_kernel forms S = X^T A X (off-diagonal ~1e-5 of its norm) and
//     eigen_finish_kernel, one or eight CTAs per matrix, diagonalises S by FP64 Jacobi
//     sweeps accumulated into X (quadratic convergence from there: two or
//     three sweeps) to 1e-14 of the Frobenius norm.
// A matrix whose FP64 sweeps do not converge (30 of them) sets the status
// word to TT_ERR_UNSUPPORTED.  Eigenvalues are returned in ascending order,
// as eigh returns them.  The buffers u, w and eigenvalues hold X, S / R and
// R's diagonal between the steps, so the call needs no workspace.
#include <math.h>

#include <cooperative_groups.h>

#include <algorithm>
#include <string>

#include "../../include/torchtree_gb300.h"
#include "tt_gamma.cuh"
#include "tt_launch.h"

namespace tt {

namespace {

constexpr int kEigMax = 64;      // largest state count
constexpr int kEigLd = kEigMax + 1;
constexpr int kEigThreads = 256;
constexpr int kEigRows = 4;  // rows of the FP64 products per CTA

// pair i of round r in the round-robin over m players (m even): player m-1
// stays, the others rotate
__device__ __forceinline__ void rr_pair(int r, int i, int m, int &p, int &q) {
  if (i == 0) {
    p = r;
    q = m - 1;
  } else {
    p = r + i < m - 1 ? r + i : r + i - (m - 1);
    q = r >= i ? r - i : r - i + (m - 1);
  }
  if (p > q) {
    const int t = p;
    p = q;
    q = t;
  }
}

// The Jacobi rotation (c, s) that zeroes a_pq of [[a_pp, a_pq], [a_pq, a_qq]]
// in FP64.  FP64 division and square root are long dependency chains on this
// GPU, and every round waits for its rotations: the angle to FP32 accuracy (a
// slightly inexact angle leaves a residual the next sweep removes), then
// c = (1 + t^2)^-1/2 from an FP32 seed by two Newton steps y <- y (3 - x y^2) / 2
// in FP64, so that c^2 + s^2 = 1 to FP64 rounding and the rotation stays
// orthogonal.  a_pq != 0.
__device__ __forceinline__ void jacobi_rotation_f64(double app, double aqq, double apq, double &c, double &s) {
  c = 1.0;
  s = 0.0;
  if (apq == 0.0) return;
  const float tf = float(aqq - app) / float(2.0 * apq);
  float t32;
  if (!(fabsf(tf) <= 1e18f)) t32 = 0.5f / tf;
  else t32 = (tf >= 0.0f ? 1.0f : -1.0f) / (fabsf(tf) + sqrtf(1.0f + tf * tf));
  const double t = double(t32), x = 1.0 + t * t;
  double y = double(rsqrtf(float(x)));
  y = y * (1.5 - 0.5 * x * y * y);
  y = y * (1.5 - 0.5 * x * y * y);
  c = y;
  s = t * y;
}

// Cyclic Jacobi sweeps on A (n x n, leading dimension NMAX + 1) accumulating
// the rotations into V, in T arithmetic, until the off-diagonal norm squared
// is at most tol2 times the Frobenius norm squared; true when converged within
// max_sweeps.  cs and pq hold a round's rotations and pairs.  Called by the
// whole CTA, of NT threads; n <= NMAX, rows NMAX + 1 apart.
template <typename T, int NMAX = kEigMax, int NT = kEigThreads>
__device__ bool jacobi_sweeps(T *A, T *V, T *cs, int *pq, double *red, int *flag, int n, double tol2,
                              int max_sweeps) {
  constexpr int NW = NT / 32, LD = NMAX + 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = n + (n & 1);  // an odd n gets a dummy player that never rotates
  const int npairs = m / 2;
  for (int sweep = 0; sweep <= max_sweeps; ++sweep) {
    // convergence: off-diagonal norm against the Frobenius norm
    double off = 0.0, tot = 0.0;
    for (int i = warp; i < n; i += NW)
      for (int j = lane; j < n; j += 32) {
        const double v = double(A[i * LD + j]);
        tot += v * v;
        if (i != j) off += v * v;
      }
    for (int o = 16; o; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      tot += __shfl_xor_sync(0xffffffffu, tot, o);
    }
    if (lane == 0) {
      red[warp] = off;
      red[NW + warp] = tot;
    }
    __syncthreads();
    if (tid == 0) {
      double so = 0.0, st = 0.0;
      for (int w = 0; w < NW; ++w) {
        so += red[w];
        st += red[NW + w];
      }
      *flag = !(so > tol2 * st) || n == 1;
    }
    __syncthreads();
    if (*flag) return true;
    if (sweep == max_sweeps) return false;
    for (int r = 0; r < m - 1; ++r) {
      // this round's pairs and rotations
      if (tid < npairs) {
        int p, qq;
        rr_pair(r, tid, m, p, qq);
        T c = T(1), s = T(0);
        if (qq < n) {
          const T apq = A[p * LD + qq];
          if (apq != T(0)) {
            if constexpr (sizeof(T) == 4) {
              const T tau = (A[qq * LD + qq] - A[p * LD + p]) / (T(2) * apq);
              T t;
              if (fabs(tau) > T(1e18)) t = T(0.5) / tau;
              else t = (tau >= T(0) ? T(1) : T(-1)) / (fabs(tau) + sqrt(T(1) + tau * tau));
              c = T(1) / sqrt(T(1) + t * t);
              s = t * c;
            } else {
              double cd, sd;
              jacobi_rotation_f64(A[p * LD + p], A[qq * LD + qq], apq, cd, sd);
              c = T(cd);
              s = T(sd);
            }
          }
        }
        cs[2 * tid] = c;
        cs[2 * tid + 1] = s;
        pq[2 * tid] = p;
        pq[2 * tid + 1] = qq;
      }
      __syncthreads();
      // rows: A <- J^T A (rows p, q of every pair), a warp per pair, lanes
      // along the row.  Distinct pairs touch distinct rows, so all of a
      // thread's loads go first (independent shared-memory latencies).
      {
        constexpr int PK = (NMAX / 2 + NW - 1) / NW;  // pairs per warp
        constexpr int HC = (NMAX + 31) / 32;             // row parts per lane
        T ap[PK][HC], aq[PK][HC], cr[PK], sr[PK];
        int pr[PK], qr[PK];
#pragma unroll
        for (int k = 0; k < PK; ++k) {
          const int i = warp + k * NW;
          pr[k] = i < npairs ? pq[2 * i] : 0;
          qr[k] = i < npairs ? pq[2 * i + 1] : n;
          cr[k] = i < npairs ? cs[2 * i] : T(1);
          sr[k] = i < npairs ? cs[2 * i + 1] : T(0);
#pragma unroll
          for (int h = 0; h < HC; ++h) {
            const int j = lane + 32 * h;
            const bool go = qr[k] < n && sr[k] != T(0) && j < n;  // not the dummy player nor the identity
            ap[k][h] = go ? A[pr[k] * LD + j] : T(0);
            aq[k][h] = go ? A[qr[k] * LD + j] : T(0);
          }
        }
#pragma unroll
        for (int k = 0; k < PK; ++k)
#pragma unroll
          for (int h = 0; h < HC; ++h) {
            const int j = lane + 32 * h;
            if (qr[k] < n && sr[k] != T(0) && j < n) {
              A[pr[k] * LD + j] = cr[k] * ap[k][h] - sr[k] * aq[k][h];
              A[qr[k] * LD + j] = sr[k] * ap[k][h] + cr[k] * aq[k][h];
            }
          }
      }
      __syncthreads();
      // columns: A <- A J, V <- V J, a warp per row, lanes over the pairs
      {
        constexpr int RK = (NMAX + NW - 1) / NW;  // rows per warp
        const int i = lane;                           // npairs <= 32
        const int pc = i < npairs ? pq[2 * i] : 0, qc = i < npairs ? pq[2 * i + 1] : n;
        const T c = i < npairs ? cs[2 * i] : T(1), s = i < npairs ? cs[2 * i + 1] : T(0);
        const bool go = qc < n && s != T(0);
        T a0[RK], a1[RK], v0[RK], v1[RK];
#pragma unroll
        for (int k = 0; k < RK; ++k) {
          const int row = warp + k * NW;
          const bool g = go && row < n;
          a0[k] = g ? A[row * LD + pc] : T(0);
          a1[k] = g ? A[row * LD + qc] : T(0);
          v0[k] = g ? V[row * LD + pc] : T(0);
          v1[k] = g ? V[row * LD + qc] : T(0);
        }
#pragma unroll
        for (int k = 0; k < RK; ++k) {
          const int row = warp + k * NW;
          if (go && row < n) {
            A[row * LD + pc] = c * a0[k] - s * a1[k];
            A[row * LD + qc] = s * a0[k] + c * a1[k];
            V[row * LD + pc] = c * v0[k] - s * v1[k];
            V[row * LD + qc] = s * v0[k] + c * v1[k];
          }
        }
      }
      __syncthreads();
    }
  }
  return false;
}

// sqrt(pi) of matrix b into sq, then A = Pi^1/2 Q Pi^-1/2 from the lower
// triangle (mirrored) into A (leading dimension kEigLd) as T; whole CTA.
template <typename T, int NMAX = kEigMax, int NT = kEigThreads>
__device__ void load_symmetrised(const double *q, const double *pi, int b, int n, double *sq, T *A) {
  constexpr int NW = NT / 32, LD = NMAX + 1;
  const double *qb = q + size_t(b) * n * n;
  for (int i = threadIdx.x; i < n; i += NT) sq[i] = sqrt(pi[size_t(b) * n + i]);
  __syncthreads();
  for (int i = threadIdx.x >> 5; i < n; i += NW)
    for (int j = threadIdx.x & 31; j < n; j += 32) {
      const int r = i >= j ? i : j, c = i >= j ? j : i;
      A[i * LD + j] = T(sq[r] * qb[r * n + c] / sq[c]);
    }
  __syncthreads();
}

// A round of the sweeps below, of m players (m even): pair i is player a = r + i and
// player b = r - i mod m - 1, pair 0 player r and player m - 1; p < q are the two.
// advance() goes to the next round.
struct EigPair {
  int a, b, p, q;
  __device__ __forceinline__ EigPair() : a(0), b(0), p(0), q(0) {}
  __device__ __forceinline__ EigPair(int i, int m) : a(i), b(i ? m - 1 - i : m - 1) { sort(); }
  __device__ __forceinline__ void sort() {
    p = min(a, b);
    q = max(a, b);
  }
  __device__ __forceinline__ void advance(int i, int m) {
    a = a + 1 == m - 1 ? 0 : a + 1;
    if (i) b = b + 1 == m - 1 ? 0 : b + 1;
    sort();
  }
};
// (u, v) <- (c u - s v, s u + c v), rounded alike wherever it is inlined: a matrix's
// system does not depend on the number of CTAs
__device__ __forceinline__ void eig_mix(float2 cs, float &u, float &v) {
  const float a = __fmaf_rn(cs.x, u, -__fmul_rn(cs.y, v)), b = __fmaf_rn(cs.y, u, __fmul_rn(cs.x, v));
  u = a;
  v = b;
}

// Step 1, a cluster of C CTAs per matrix: FP32 Jacobi sweeps on A until the
// off-diagonal norm is below 1e-6 of the Frobenius norm (at most kEigStartSweeps:
// FP32 rounding may stop short of that); the eigenvector matrix X0, in FP64, into
// x.  The first CTA rotates A alone: of the blocks of four elements that two
// rotations of a round mix, a thread holds one or two (rows first, columns then;
// each element belongs to one block, so a round takes two barriers and one pass over
// A), and every CTA's shared memory is given the rotations.  A row of X0 is the unit
// row under all the rotations, whatever the other rows do: afterwards each warp
// carries its rows through them in registers, a pair per lane, the players moving
// from lane to lane as the round-robin does.  Bound by the latency of a round (the
// rotation's divisions and roots, two barriers).  61 states, 6 x 61 rounds: 534 us
// with separate passes over rows and columns and X0 rotated along, 336 us so;
// 20 states 119 -> 64 us, the same rotations and bits.
constexpr int kEigStartSweeps = 6;

template <int NMAX>
constexpr int eig_start_threads() { return NMAX == 64 ? 512 : 256; }
template <int NMAX>
constexpr size_t eig_start_smem() {  // A and all rounds' rotations
  return (size_t(NMAX) * (NMAX + 1) + 2 * size_t(kEigStartSweeps) * (NMAX - 1) * (NMAX / 2)) * sizeof(float);
}

template <int NMAX, int C>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(eig_start_threads<NMAX>())
    eigen_start_kernel(const double *q, const double *pi, int n, double *x) {
  namespace cg = cooperative_groups;
  constexpr int NT = eig_start_threads<NMAX>(), NW = NT / 32, LD = NMAX + 1, H = NMAX / 2;
  constexpr int RPW = (NMAX + C * NW - 1) / (C * NW);  // rows of X0 per warp
  constexpr int BPT = H * H / NT;                      // blocks per thread
  extern __shared__ __align__(16) float esm[];
  float2 *log = reinterpret_cast<float2 *>(esm);                  // [round][npairs] (c, s)
  float *A = esm + 2 * kEigStartSweeps * (NMAX - 1) * H;          // [n + 1][LD], a zero dummy player
  __shared__ double red[2 * NW], sq[NMAX];
  __shared__ int flag, rounds;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = C > 1 ? int(cluster.block_rank()) : 0;
  const int b = blockIdx.x / C, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = n + (n & 1), npairs = m / 2;
  if constexpr (C > 1) cluster.sync();  // every CTA runs before the first one writes to it
  if (rank == 0) {
    load_symmetrised<float, NMAX, NT>(q, pi, b, n, sq, A);
    if (n < m)
      for (int k = tid; k < m; k += NT) A[n * LD + k] = A[k * LD + n] = 0.0f;
    // this thread's blocks: a pair of columns, BPT pairs of rows
    const int bj = tid % H, bi = tid / H;
    EigPair pj(min(bj, npairs - 1), m), pr[BPT];
#pragma unroll
    for (int k = 0; k < BPT; ++k) pr[k] = EigPair(min(bi + k * (NT / H), npairs - 1), m);
    __syncthreads();
    int done = 0;
    for (int sweep = 0; sweep <= kEigStartSweeps; ++sweep) {
      double off = 0.0, tot = 0.0;
      for (int i = warp; i < n; i += NW)
        for (int j = lane; j < n; j += 32) {
          const double v = double(A[i * LD + j]);
          tot += v * v;
          if (i != j) off += v * v;
        }
      for (int o = 16; o; o >>= 1) {
        off += __shfl_xor_sync(0xffffffffu, off, o);
        tot += __shfl_xor_sync(0xffffffffu, tot, o);
      }
      if (lane == 0) {
        red[warp] = off;
        red[NW + warp] = tot;
      }
      __syncthreads();
      if (tid == 0) {
        double so = 0.0, st = 0.0;
        for (int w = 0; w < NW; ++w) {
          so += red[w];
          st += red[NW + w];
        }
        flag = !(so > 1e-12 * st);
      }
      __syncthreads();
      if (flag || sweep == kEigStartSweeps) break;
      for (int r = 0; r < m - 1; ++r, ++done) {
        if (tid < npairs) {  // this round's rotations
          const float apq = A[pj.p * LD + pj.q];
          float c = 1.0f, sn = 0.0f;
          if (apq != 0.0f) {
            const float tau = (A[pj.q * (LD + 1)] - A[pj.p * (LD + 1)]) / (2.0f * apq);
            float t;
            if (fabsf(tau) > 1e18f) t = 0.5f / tau;
            else t = (tau >= 0.0f ? 1.0f : -1.0f) / (fabsf(tau) + sqrtf(__fmaf_rn(tau, tau, 1.0f)));
            c = 1.0f / sqrtf(__fmaf_rn(t, t, 1.0f));
            sn = t * c;
          }
          const float2 cs = make_float2(c, sn);
          log[done * npairs + tid] = cs;
#pragma unroll
          for (int o = 1; o < C; ++o) cluster.map_shared_rank(log, o)[done * npairs + tid] = cs;
        }
        __syncthreads();
        if (bj < npairs) {
          const float2 rj = log[done * npairs + bj];
#pragma unroll
          for (int k = 0; k < BPT; ++k) {
            const int i = bi + k * (NT / H);
            if (i >= npairs) continue;
            const float2 ri = log[done * npairs + i];
            float *Ap = A + pr[k].p * LD, *Aq = A + pr[k].q * LD;
            float a0 = Ap[pj.p], a1 = Ap[pj.q], b0 = Aq[pj.p], b1 = Aq[pj.q];
            eig_mix(ri, a0, b0);  // rows
            eig_mix(ri, a1, b1);
            eig_mix(rj, a0, a1);  // columns
            eig_mix(rj, b0, b1);
            Ap[pj.p] = a0;
            Ap[pj.q] = a1;
            Aq[pj.p] = b0;
            Aq[pj.q] = b1;
            pr[k].advance(i, m);
          }
        }
        pj.advance(bj, m);
        __syncthreads();
      }
    }
    if (tid == 0) {
      rounds = done;
#pragma unroll
      for (int o = 1; o < C; ++o) *cluster.map_shared_rank(&rounds, o) = done;
    }
  }
  if constexpr (C > 1) cluster.sync();
  else __syncthreads();
  // rows of X0: lane i carries the columns of pair i
  const int total = rounds, last = npairs - 1;
  EigPair at(lane, m);
  const int row0 = (rank * NW + warp) * RPW;
  if (row0 >= n) return;  // a whole warp; nothing reaches into this CTA any more
  float va[RPW], vb[RPW];
#pragma unroll
  for (int k = 0; k < RPW; ++k) {
    va[k] = lane <= last && at.a == row0 + k ? 1.0f : 0.0f;
    vb[k] = lane <= last && at.b == row0 + k ? 1.0f : 0.0f;
  }
  const float2 *cs = log + min(lane, last);
  for (int d = 0; d < total; ++d, cs += npairs) {
    const float2 rot = *cs;
    const bool swap = at.a > at.b;
#pragma unroll
    for (int k = 0; k < RPW; ++k) {
      float vp = swap ? vb[k] : va[k], vq = swap ? va[k] : vb[k];
      eig_mix(rot, vp, vq);
      const float na = swap ? vq : vp, nb = swap ? vp : vq;
      // the next round's pairs: p from the lane above (the last lane's is its q), q from the lane
      // below (lane 1's is lane 0's p); player m - 1 stays in lane 0
      const float da = __shfl_down_sync(0xffffffffu, na, 1);
      const float ub = __shfl_up_sync(0xffffffffu, lane == 0 ? na : nb, 1);
      va[k] = lane == last ? nb : da;
      vb[k] = lane == 0 ? nb : ub;
    }
    at.advance(lane, m);
  }
  double *xb = x + size_t(b) * n * n;
  if (lane <= last) {
#pragma unroll
    for (int k = 0; k < RPW; ++k)
      if (row0 + k < n) {
        xb[(row0 + k) * n + at.a] = double(va[k]);
        if (at.b < n) xb[(row0 + k) * n + at.b] = double(vb[k]);
      }
  }
}

// Step 2 / 3, kEigRows rows per CTA (grid: row blocks x matrices), FP64: for
// the current eigenvector estimate X (x),
//   R = I - X^T X   (strict lower triangle into w, diagonal into lam),
//   S = X^T A X     (upper triangle with the diagonal into w; with_s only).
// Both are symmetric, so one n x n buffer holds the two.
__global__ void __launch_bounds__(kEigThreads) eigen_gram_kernel(const double *q, const double *pi, int n,
                                                                 const double *x, double *w, double *lam,
                                                                 int with_s) {
  constexpr int NW = kEigThreads / 32;
  extern __shared__ __align__(16) double gsm[];
  double *A = gsm;                      // [n][kEigLd]
  double *X = A + kEigMax * kEigLd;     // [n][kEigLd]
  double *M = X + kEigMax * kEigLd;     // [kEigRows][kEigLd]: rows of X^T A
  double *sq = M + kEigRows * kEigLd;   // [n]
  const int b = blockIdx.y, i0 = blockIdx.x * kEigRows, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rows = min(kEigRows, n - i0);
  const double *xb = x + size_t(b) * n * n;
  for (int i = warp; i < n; i += NW)
    for (int j = lane; j < n; j += 32) X[i * kEigLd + j] = xb[i * n + j];
  if (with_s) load_symmetrised(q, pi, b, n, sq, A);
  else __syncthreads();
  double *wb = w + size_t(b) * n * n;
  // R rows i0 .. i0 + rows - 1, columns j <= i; two warps per row
  for (int t = warp; t < 2 * rows; t += NW) {
    const int r = t >> 1, i = i0 + r;
    for (int j = (t & 1) * 32 + lane; j <= i; j += 64) {
      double s = 0.0;
      for (int k = 0; k < n; ++k) s = fma(X[k * kEigLd + i], X[k * kEigLd + j], s);
      if (j < i) wb[i * n + j] = -s;
      else lam[size_t(b) * n + i] = 1.0 - s;
    }
  }
  if (!with_s) return;
  for (int t = warp; t < 2 * rows; t += NW) {
    const int r = t >> 1, i = i0 + r;
    for (int j = (t & 1) * 32 + lane; j < n; j += 64) {
      double s = 0.0;
      for (int k = 0; k < n; ++k) s = fma(X[k * kEigLd + i], A[k * kEigLd + j], s);
      M[r * kEigLd + j] = s;
    }
  }
  __syncthreads();
  for (int t = warp; t < 2 * rows; t += NW) {
    const int r = t >> 1, i = i0 + r;
    for (int j = i + (t & 1) * 32 + lane; j < n; j += 64) {
      double s = 0.0;
      for (int k = 0; k < n; ++k) s = fma(M[r * kEigLd + k], X[k * kEigLd + j], s);
      wb[i * n + j] = s;
    }
  }
}

// Step 2, kEigRows rows per CTA, FP64: one Newton-Schulz step
// X <- X + X R / 2 = X (3I - X^T X) / 2 with R = I - X^T X from the last
// eigen_gram_kernel.  A row of the result needs only that row of X, so each
// CTA updates its own rows in place.
__global__ void __launch_bounds__(kEigThreads) eigen_orth_kernel(int n, double *x, const double *w,
                                                                 const double *lam) {
  constexpr int NW = kEigThreads / 32;
  extern __shared__ __align__(16) double osm[];
  double *R = osm;                      // [n][kEigLd], halved
  double *Xr = R + kEigMax * kEigLd;    // [kEigRows][kEigLd]
  const int b = blockIdx.y, i0 = blockIdx.x * kEigRows, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rows = min(kEigRows, n - i0);
  const double *wb = w + size_t(b) * n * n, *rd = lam + size_t(b) * n;
  double *xb = x + size_t(b) * n * n;
  for (int i = warp; i < n; i += NW)
    for (int j = lane; j < n; j += 32)
      R[i * kEigLd + j] = 0.5 * (i == j ? rd[i] : wb[max(i, j) * n + min(i, j)]);
  for (int r = warp; r < rows; r += NW)
    for (int j = lane; j < n; j += 32) Xr[r * kEigLd + j] = xb[(i0 + r) * n + j];
  __syncthreads();
  for (int t = warp; t < 2 * rows; t += NW) {
    const int r = t >> 1;
    for (int j = (t & 1) * 32 + lane; j < n; j += 64) {
      double s = Xr[r * kEigLd + j];
      for (int k = 0; k < n; ++k) s = fma(Xr[r * kEigLd + k], R[k * kEigLd + j], s);
      xb[(i0 + r) * n + j] = s;
    }
  }
}

// Step 3, a cluster of C CTAs per matrix, FP64: S = X^T A X (in W, upper
// triangle) and X (in U); FP64 Jacobi sweeps on S, accumulated into X, to 1e-14 of
// the Frobenius norm; a matrix that does not converge in 30 sweeps sets the status
// word.  Eigenvalues ascending, with U = Pi^-1/2 X and W = X^T Pi^1/2.
// Every CTA keeps a copy of A, in two buffers.  A round: every CTA
// forms the same rotations from its copy; of the blocks of four elements that two
// rotations mix, each CTA updates its share, two threads a block, a row of it each,
// rows first and columns then, and writes the results into every CTA's other buffer
// through distributed shared memory (consecutive lanes along a row: the stores that
// coalesce; the rotations of a round read the buffer that nobody writes); while they
// travel it rotates its own rows of X.  One cluster barrier a round.  Bound by FP64
// latency and arithmetic (64 cycles per warp instruction and SM quarter).  61 states:
// 1 matrix 528 -> 401 us, 16 matrices 531 -> 488 us, against 4 CTAs with full copies
// and rows and columns in separate passes.  Up to 32 states one CTA (20 states:
// 216 -> 93 us).  With the upper triangle alone (352 / 431 / 83 us) the last
// bits change, and with them the rounding of FP32 transition matrices.
constexpr int kEigCluster = 8;

template <int NMAX, int C>
constexpr size_t eig_finish_smem() {  // A twice, rows of X, rotations twice, sqrt(pi)
  return (2 * size_t(NMAX) * (NMAX + 1) + size_t((NMAX + C - 1) / C) * (NMAX + 1) + 2 * NMAX + NMAX) *
         sizeof(double);
}

template <int NMAX, int C>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(kEigThreads)
    eigen_finish_kernel(const double *pi, int n, double *lam, double *U, double *W, int *status) {
  namespace cg = cooperative_groups;
  constexpr int NT = kEigThreads, NW = NT / 32, LD = NMAX + 1, H = NMAX / 2, BUF = NMAX * LD;
  constexpr int NB = ((H * H + C - 1) / C + 31) / 32 * 32;            // this CTA's blocks, at most
  constexpr int HB = (2 * NB + NT - 1) / NT;                          // half blocks per thread
  extern __shared__ __align__(16) double fsm[];
  double *A = fsm;                                        // [2][n + 1][LD]
  double *V = A + 2 * BUF;                                // [rows][LD]: rows = rank mod C of X
  double2 *cs = reinterpret_cast<double2 *>(V + (NMAX + C - 1) / C * LD + ((NMAX + C - 1) / C * LD & 1));
  double *sq = reinterpret_cast<double *>(cs + 2 * H);    // [n]
  __shared__ double red[2 * NW];
  __shared__ int flag;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = C > 1 ? int(cluster.block_rank()) : 0;
  const int b = blockIdx.x / C, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int m = n + (n & 1), npairs = m / 2;
  const size_t mo = size_t(b) * n * n;
  for (int i = tid; i < n; i += NT) sq[i] = sqrt(pi[size_t(b) * n + i]);
  for (int i = warp; i < m; i += NW)
    for (int j = lane; j < m; j += 32) {
      A[i * LD + j] = i < n && j < n ? W[mo + size_t(min(i, j)) * n + max(i, j)] : 0.0;  // a dummy player of zeros
      if (i % C == rank) V[i / C * LD + j] = i < n && j < n ? U[mo + size_t(i) * n + j] : 0.0;
    }
  if constexpr (C > 1) cluster.sync();  // every CTA has read U and W before any writes its outputs
  else __syncthreads();
  // this thread's half blocks: pairs of rows and columns and which row of the two; its lane's pair
  int hi[HB], hj[HB];
  const int blocks = npairs * npairs, share = (blocks + C - 1) / C;
  EigPair row_pair(tid % H, m), pi_[HB], pj[HB];
#pragma unroll
  for (int k = 0; k < HB; ++k) {
    const int h = tid + k * NT, at = h < NB ? h : h - NB, e = rank * share + at;  // a warp's lanes along a row
    const bool mine = h < 2 * NB && at < share && e < blocks;
    hi[k] = mine ? e / npairs : -1;
    hj[k] = mine ? e % npairs : -1;
    if (!mine) continue;
    pi_[k] = EigPair(hi[k], m);
    pj[k] = EigPair(hj[k], m);
  }
  double *cur = A, *nxt = A + BUF;
  bool ok = false;
  for (int sweep = 0; sweep <= 30; ++sweep) {
    double off = 0.0, tot = 0.0;
    for (int i = warp; i < n; i += NW)
      for (int j = lane; j < n; j += 32) {
        const double v = cur[i * LD + j];
        tot += v * v;
        if (i != j) off += v * v;
      }
    for (int o = 16; o; o >>= 1) {
      off += __shfl_xor_sync(0xffffffffu, off, o);
      tot += __shfl_xor_sync(0xffffffffu, tot, o);
    }
    if (lane == 0) {
      red[warp] = off;
      red[NW + warp] = tot;
    }
    __syncthreads();
    if (tid == 0) {
      double so = 0.0, st = 0.0;
      for (int w = 0; w < NW; ++w) {
        so += red[w];
        st += red[NW + w];
      }
      flag = !(so > 1e-28 * st) || n == 1;
    }
    __syncthreads();
    if (flag) {
      ok = true;
      break;
    }
    if (sweep == 30) break;
    for (int r = 0; r < m - 1; ++r) {
      double2 *rot = cs + (r & 1) * H;  // the last round's may still be read
      if (tid < npairs) {  // the round's rotations, the same in every CTA
        double c, sn;
        jacobi_rotation_f64(cur[row_pair.p * (LD + 1)], cur[row_pair.q * (LD + 1)],
                            cur[row_pair.p * LD + row_pair.q], c, sn);
        rot[tid] = make_double2(c, sn);
      }
      __syncthreads();
#pragma unroll
      for (int k = 0; k < HB; ++k) {
        if (hi[k] < 0) continue;
        const double2 ri = rot[hi[k]], rj = rot[hj[k]];
        const bool second = tid + k * NT >= NB;
        const double *rp = cur + pi_[k].p * LD, *rq = cur + pi_[k].q * LD;
        const int o0 = (second ? pi_[k].q : pi_[k].p) * LD + pj[k].p, o1 = o0 + pj[k].q - pj[k].p;
        const double app = rp[pj[k].p], apq = rp[pj[k].q], aqp = rq[pj[k].p], aqq = rq[pj[k].q];
        pi_[k].advance(hi[k], m);
        pj[k].advance(hj[k], m);
        // the row of pair i: c p - s q, or s p + c q
        const double u = second ? ri.y : ri.x, w = second ? ri.x : -ri.y;
        const double x0 = u * app + w * aqp, x1 = u * apq + w * aqq;
        const double n0 = rj.x * x0 - rj.y * x1, n1 = rj.y * x0 + rj.x * x1;
        const int base = int(nxt - A);
#pragma unroll
        for (int o = 0; o < C; ++o) {
          double *dst = C > 1 ? cluster.map_shared_rank(A, o) + base : nxt;
          dst[o0] = n0;
          dst[o1] = n1;
        }
      }
      __syncwarp();
      if constexpr (C > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      // this CTA's rows of X, lanes over the pairs
      if (tid % H < npairs) {
        const double2 rl = rot[tid % H];
        for (int row = tid / H; row * C + rank < n; row += NT / H) {
          const double vp = V[row * LD + row_pair.p], vq = V[row * LD + row_pair.q];
          V[row * LD + row_pair.p] = rl.x * vp - rl.y * vq;
          V[row * LD + row_pair.q] = rl.y * vp + rl.x * vq;
        }
      }
      row_pair.advance(tid % H, m);
      __syncwarp();
      if constexpr (C > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
      else __syncthreads();
      double *t = cur;
      cur = nxt;
      nxt = t;
    }
  }
  if (tid == 0 && rank == 0 && !ok) atomicExch(status, TT_ERR_UNSUPPORTED);
  __syncthreads();
  // ascending order: the rank of each eigenvalue (ties by index); this CTA's rows of U and W
  for (int k = tid; k < n; k += NT) {
    const double lk = cur[k * LD + k];
    int rk = 0;
    for (int j = 0; j < n; ++j) {
      const double lj = cur[j * LD + j];
      rk += lj < lk || (lj == lk && j < k);
    }
    if (rank == 0) lam[size_t(b) * n + rk] = lk;
    for (int i = rank; i < n; i += C) {
      U[(size_t(b) * n + i) * n + rk] = V[i / C * LD + k] / sq[i];  // U = Pi^-1/2 V
      W[(size_t(b) * n + rk) * n + i] = V[i / C * LD + k] * sq[i];  // W = V^T Pi^1/2
    }
  }
}

__global__ void __launch_bounds__(32) gamma_quantiles_kernel(const double *shape, int K, double *x, double *dxda) {
  const int e = blockIdx.x, b = e / K, k = e - b * K;
  const double q = (2.0 * k + 1.0) / (2.0 * K);
  double xv = 0.0, dv = 0.0;
  if (!gamma_quantile_warp(shape[b], q, xv, dv)) xv = dv = __longlong_as_double(0x7ff8000000000000ll);  // NaN
  if (threadIdx.x == 0) {
    x[e] = xv;
    dxda[e] = dv;
  }
}

// Matrices of at most kEigSmall states: the three steps above in one launch, a warp
// per matrix, with their arithmetic.  At 4 states each of the seven launches is a few
// microseconds of one CTA, mostly barriers of eight warps: 52 -> 34 us and six
// launches fewer.
constexpr int kEigSmall = 4;

__global__ void __launch_bounds__(32) eigen_small_kernel(const double *q, const double *pi, int n, double *lam,
                                                         double *U, double *W, int *status) {
  constexpr int N = kEigSmall, LD = N + 1;
  __shared__ float Af[N * LD], Vf[N * LD], csf[N];
  __shared__ double A[N * LD], X[N * LD], R[N * LD], M[N * LD], cs[N], red[2], sq[N];
  __shared__ int pq[N], flag;
  const int b = blockIdx.x, lane = threadIdx.x;
  load_symmetrised<float, N, 32>(q, pi, b, n, sq, Af);
  for (int e = lane; e < n * n; e += 32) Vf[e / n * LD + e % n] = e / n == e % n ? 1.0f : 0.0f;
  __syncthreads();
  jacobi_sweeps<float, N, 32>(Af, Vf, csf, pq, red, &flag, n, 1e-12, 6);
  for (int e = lane; e < n * n; e += 32) X[e / n * LD + e % n] = double(Vf[e / n * LD + e % n]);
  load_symmetrised<double, N, 32>(q, pi, b, n, sq, A);
  const int i = lane / N, j = lane % N;  // lanes 0-15: an entry each
  const bool in = i < n && j < n;
  for (int it = 0; it < 2; ++it) {  // X <- X + X R / 2, R = I - X^T X
    if (in && j <= i) {
      double s = 0.0;
      for (int k = 0; k < n; ++k) s = fma(X[k * LD + i], X[k * LD + j], s);
      R[i * LD + j] = 0.5 * (j < i ? -s : 1.0 - s);
    }
    __syncthreads();
    double s = 0.0;
    if (in) {
      s = X[i * LD + j];
      for (int k = 0; k < n; ++k) s = fma(X[i * LD + k], R[max(k, j) * LD + min(k, j)], s);
    }
    __syncthreads();
    if (in) X[i * LD + j] = s;
    __syncthreads();
  }
  if (in) {  // S = X^T A X, upper triangle mirrored
    double s = 0.0;
    for (int k = 0; k < n; ++k) s = fma(X[k * LD + i], A[k * LD + j], s);
    M[i * LD + j] = s;
  }
  __syncthreads();
  if (in && j >= i) {
    double s = 0.0;
    for (int k = 0; k < n; ++k) s = fma(M[i * LD + k], X[k * LD + j], s);
    A[i * LD + j] = s;
    A[j * LD + i] = s;
  }
  __syncthreads();
  const bool ok = jacobi_sweeps<double, N, 32>(A, X, cs, pq, red, &flag, n, 1e-28, 30);
  if (lane == 0 && !ok) atomicExch(status, TT_ERR_UNSUPPORTED);
  if (in) {  // eigenvalue j goes to its rank (ties by index)
    const double lj = A[j * LD + j];
    int rank = 0;
    for (int k = 0; k < n; ++k) {
      const double lk = A[k * LD + k];
      rank += lk < lj || (lk == lj && k < j);
    }
    if (i == 0) lam[size_t(b) * n + rank] = lj;
    U[(size_t(b) * n + i) * n + rank] = X[i * LD + j] / sq[i];
    W[(size_t(b) * n + rank) * n + i] = X[i * LD + j] * sq[i];
  }
}

int efail(int code, const std::string &msg) { return record_error(code, msg.c_str()); }

}  // namespace

}  // namespace tt

extern "C" {

int tt_reversible_eigen(int32_t batch, int32_t state_count, const double *q, const double *frequencies,
                        double *eigenvalues, double *u, double *w, int32_t *status, void *stream) {
  if (!q || !frequencies || !eigenvalues || !u || !w || !status)
    return tt::efail(TT_ERR_INVALID_ARGUMENT, "NULL argument");
  if (batch < 1 || state_count < 1 || state_count > tt::kEigMax)
    return tt::efail(TT_ERR_INVALID_ARGUMENT, "tt_reversible_eigen: batch >= 1 and 1 <= state_count <= 64");
  using namespace tt;
  const int n = state_count;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const size_t gram_smem = (2 * size_t(kEigMax) * kEigLd + kEigRows * kEigLd + kEigMax) * sizeof(double);
  const size_t orth_smem = (size_t(kEigMax) * kEigLd + kEigRows * kEigLd) * sizeof(double);
  if (n <= kEigSmall) {
    eigen_small_kernel<<<batch, 32, 0, s>>>(q, frequencies, n, eigenvalues, u, w, status);
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TT_OK : tt::efail(TT_ERR_CUDA, std::string("eigen launch: ") + cudaGetErrorString(e));
  }
  cudaError_t e = kernel_smem(eigen_gram_kernel, gram_smem);
  if (e == cudaSuccess) e = kernel_smem(eigen_orth_kernel, orth_smem);
  if (e == cudaSuccess) e = kernel_smem(eigen_start_kernel<64, 4>, eig_start_smem<64>());
  if (e == cudaSuccess) e = kernel_smem(eigen_start_kernel<64, 1>, eig_start_smem<64>());
  if (e == cudaSuccess) e = kernel_smem(eigen_finish_kernel<64, kEigCluster>, eig_finish_smem<64, kEigCluster>());
  // matrices in groups of at most 65,535 (the grid's y extent of the row-block kernels)
  for (int b0 = 0; e == cudaSuccess && b0 < batch; b0 += 65535) {
    const int nb = std::min(batch - b0, 65535);
    const size_t mo = size_t(b0) * n * n, vo = size_t(b0) * n;
    const double *qb = q + mo, *pib = frequencies + vo;
    double *ub = u + mo, *wb = w + mo, *lb = eigenvalues + vo;
    const dim3 rows_grid((n + kEigRows - 1) / kEigRows, nb);
    if (n <= 32) {
      eigen_start_kernel<32, 1><<<nb, eig_start_threads<32>(), eig_start_smem<32>(), s>>>(qb, pib, n, ub);
    } else if (nb <= 76) {  // four CTAs each while 152 SMs hold them at two CTAs per SM (64 matrices 443 us);
                            // more take one each (300 matrices 516 us, 719 before)
      eigen_start_kernel<64, 4><<<4 * nb, eig_start_threads<64>(), eig_start_smem<64>(), s>>>(qb, pib, n, ub);
    } else {
      eigen_start_kernel<64, 1><<<nb, eig_start_threads<64>(), eig_start_smem<64>(), s>>>(qb, pib, n, ub);
    }
    for (int it = 0; it < 2; ++it) {
      eigen_gram_kernel<<<rows_grid, kEigThreads, gram_smem, s>>>(qb, pib, n, ub, wb, lb, 0);
      eigen_orth_kernel<<<rows_grid, kEigThreads, orth_smem, s>>>(n, ub, wb, lb);
    }
    eigen_gram_kernel<<<rows_grid, kEigThreads, gram_smem, s>>>(qb, pib, n, ub, wb, lb, 1);
    if (n > 32)
      eigen_finish_kernel<64, kEigCluster><<<nb * kEigCluster, kEigThreads, eig_finish_smem<64, kEigCluster>(), s>>>(
          pib, n, lb, ub, wb, status);
    else
      eigen_finish_kernel<32, 1><<<nb, kEigThreads, eig_finish_smem<32, 1>(), s>>>(pib, n, lb, ub, wb, status);
    e = cudaGetLastError();
  }
  return e == cudaSuccess ? TT_OK : tt::efail(TT_ERR_CUDA, std::string("eigen launch: ") + cudaGetErrorString(e));
}

int tt_gamma_quantiles(int32_t batch, int32_t category_count, const double *shape, double *x, double *dx_dshape,
                       void *stream) {
  if (!shape || !x || !dx_dshape) return tt::efail(TT_ERR_INVALID_ARGUMENT, "NULL argument");
  if (batch < 1 || category_count < 1) return tt::efail(TT_ERR_INVALID_ARGUMENT, "batch and categories must be >= 1");
  const int n = batch * category_count;
  // one warp per quantile and per CTA: the FP64 work spreads over as many SMs as there are quantiles
  tt::gamma_quantiles_kernel<<<n, 32, 0, static_cast<cudaStream_t>(stream)>>>(shape, category_count, x, dx_dshape);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? TT_OK
                          : tt::efail(TT_ERR_CUDA, std::string("gamma quantile launch: ") + cudaGetErrorString(e));
}

int tt_gamma_quantiles_host(int32_t batch, int32_t category_count, const double *shape, double *x,
                            double *dx_dshape) {
  if (!shape || !x || !dx_dshape) return tt::efail(TT_ERR_INVALID_ARGUMENT, "NULL argument");
  if (batch < 1 || category_count < 1) return tt::efail(TT_ERR_INVALID_ARGUMENT, "batch and categories must be >= 1");
  for (int b = 0; b < batch; ++b)
    for (int k = 0; k < category_count; ++k) {
      const double q = (2.0 * k + 1.0) / (2.0 * category_count);
      if (!tt::gamma_quantile(shape[b], q, x[b * category_count + k], dx_dshape[b * category_count + k]))
        return tt::efail(TT_ERR_INVALID_ARGUMENT, "Gamma quantile: the shape must be finite and > 0");
    }
  return TT_OK;
}

}  // extern "C"
