// The small per-call pieces around the pruning passes, each one launch where
// tensor operations took ten to thirty: category rates with their shape
// derivative, rate matrices from exchangeabilities, and a whole evaluation
// (normalised rate matrix, eigen system, transition matrices, post-order) and
// its gradient behind one call each.
//
// A log-likelihood with gradient at 69 taxa x 238 patterns runs 0.25 ms of
// pruning kernels; as separate tensor operations the model set-up and its
// backward were 80 more launches and 1.9 ms of host time (98 launches, 1,932 us per
// call -> 20 launches, 612 us; value only at 137 taxa 660 -> 212 us).  The kernels here
// are bound by launch latency (one CTA per sample, a few microseconds), so
// they are written for few dependent steps, not for throughput.
#include <algorithm>
#include <cstring>
#include <string>

#include "../../include/torchtree_gb300.h"
#include "tt_common.cuh"
#include "tt_gamma.cuh"
#include "tt_launch.h"
#include "tt_plan.h"

namespace tt {
namespace {

int sfail(int code, const std::string &m) { return record_error(code, m.c_str()); }
int sdone(cudaError_t e, const char *what) {
  return e == cudaSuccess ? TT_OK : sfail(TT_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ double lane_sum(double v) {  // the same bits in every lane
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kAll, v, o);
  return v;
}

// term(0) + .. + term(n - 1) in the order in which the tensor compositions' row sums run
// (L = the largest power of two up to 32 that is at most n: lane l takes l, l + L, ..; then
// pairs of neighbours, of neighbouring pairs, ..), in every lane: rates and rate matrices
// keep the compositions' bits, which FP32 transition matrices are rounded from.
template <typename F>
__device__ __forceinline__ double row_sum(int n, F term) {
  const int lane = threadIdx.x & 31, L = n >= 32 ? 32 : 1 << (31 - __clz(n));
  double s = 0.0;
  if (lane < L)
    for (int j = lane; j < n; j += L) s = __dadd_rn(s, term(j));
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) s = __dadd_rn(s, __shfl_down_sync(kAll, s, o));
  return __shfl_sync(kAll, s, 0);
}

// Mean-one rates and their shape derivative from lane k's raw rate r and dr
// (one warp, lanes >= K zero); equal category weights 1 / K.
__device__ __forceinline__ void finish_rates(double r, double dr, int K, int b, double *rates, double *drates,
                                             double *probs) {
  const int k = threadIdx.x & 31;
  const double w = 1.0 / K, dm = lane_sum(dr * w);
  __shared__ double rw[32];
  rw[k] = __dmul_rn(r, w);
  __syncwarp();
  const double m = row_sum(K, [&](int j) { return rw[j]; });
  if (k < K) {
    const double rho = r / m;
    rates[size_t(b) * K + k] = rho;
    drates[size_t(b) * K + k] = (dr - rho * dm) / m;
    if (b == 0) probs[k] = w;
  }
}

__global__ void __launch_bounds__(32) weibull_rates_kernel(const double *shape, int K, double *rates, double *drates,
                                                           double *probs) {
  const int b = blockIdx.x, k = threadIdx.x;
  double r = 0.0, dr = 0.0;
  if (k < K) {
    // (a tensor over a number is multiplied by the number's reciprocal)
    const double q = __dmul_rn(2.0 * k + 1.0, 1.0 / (2.0 * K)), x = -log(1.0 - q), inv = 1.0 / shape[b];
    r = pow(x, inv);
    dr = -r * log(x) * inv * inv;
  }
  finish_rates(r, dr, K, b, rates, drates, probs);
}

// a CTA per sample, a warp per quantile (the first 8 at once)
__global__ void __launch_bounds__(256) gamma_rates_kernel(const double *shape, int K, double *rates, double *drates,
                                                          double *probs) {
  __shared__ double xs[32], ds[32];
  const int b = blockIdx.x, lane = threadIdx.x & 31;
  const double a = shape[b];
  for (int k = threadIdx.x >> 5; k < K; k += blockDim.x >> 5) {
    double x = 0.0, d = 0.0;
    if (!gamma_quantile_warp(a, (2.0 * k + 1.0) / (2.0 * K), x, d)) x = d = __longlong_as_double(0x7ff8000000000000ll);
    if (lane == 0) xs[k] = x, ds[k] = d;
  }
  __syncthreads();
  if (threadIdx.x >= 32) return;
  const double r = lane < K ? xs[lane] / a : 0.0, dr = lane < K ? ds[lane] / a - xs[lane] / (a * a) : 0.0;
  finish_rates(r, dr, K, b, rates, drates, probs);
}

__global__ void __launch_bounds__(32) rates_backward_kernel(const double *grad, const double *drates, int K,
                                                            double *dshape) {
  const int b = blockIdx.x, k = threadIdx.x;
  const double s = lane_sum(k < K ? grad[size_t(b) * K + k] * drates[size_t(b) * K + k] : 0.0);
  if (k == 0) dshape[b] = s;
}

// ------------------------------------------------------------ rate matrices
// Exchangeability of upper-triangle entry e: the parameter of that index, or
// with a map the product of up to two of the (at most three) parameters.
// The map travels as a kernel parameter (at most 4,032 bytes), so no device copy
// of it has to be kept anywhere.
struct NoMap {};
struct PairMap {
  static constexpr int kWords = 2 * 64 * 63 / 2 / 4;
  uint32_t m[kWords];  // [2][S (S-1) / 2] parameter indices (-1: 1), four to a word
};

template <typename Map>
struct Exch {
  static constexpr bool kMapped = sizeof(Map) > 1;
  const double *p[3];
  int n[3];
  int count;  // S (S-1) / 2
  Map map;
  __device__ __forceinline__ double param(int b, int i) const {
    if (i < 0) return 1.0;
    if (i < n[0]) return p[0][size_t(b) * n[0] + i];
    i -= n[0];
    if (i < n[1]) return p[1][size_t(b) * n[1] + i];
    return p[2][size_t(b) * n[2] + i - n[1]];
  }
  // the map into shared memory: a parameter indexed per lane is read one lane at a time (with
  // the pairs read from it directly, 118 us at 61 states)
  __device__ __forceinline__ const int8_t *stage(uint32_t *sm) const {
    if constexpr (kMapped) {
      for (int w = threadIdx.x; w < PairMap::kWords; w += blockDim.x) sm[w] = map.m[w];
      __syncthreads();
    }
    return reinterpret_cast<const int8_t *>(sm);
  }
  // (plus 0: the composition adds the upper triangle to a transposed one of zeros, so no -0)
  __device__ __forceinline__ double value(int b, const int8_t *m, int e) const {
    if constexpr (kMapped) return __dadd_rn(__dmul_rn(param(b, m[e]), param(b, m[count + e])), 0.0);
    else return __dadd_rn(p[0][size_t(b) * n[0] + e], 0.0);
  }
};

__device__ __forceinline__ int upper_index(int i, int j, int S) {  // i != j
  const int a = min(i, j), c = max(i, j);
  return a * S - a * (a + 1) / 2 + c - a - 1;
}

template <typename Map>
__global__ void __launch_bounds__(256) exch_q_kernel(const __grid_constant__ Exch<Map> x, const double *pi, int S, double *q) {
  __shared__ uint32_t sm[Exch<Map>::kMapped ? PairMap::kWords : 1];
  const int8_t *m = x.stage(sm);
  const int b = blockIdx.x;
  const double *pb = pi + size_t(b) * S;
  double *qb = q + size_t(b) * S * S;
  for (int e = threadIdx.x; e < S * S; e += blockDim.x) {
    const int i = e / S, j = e - i * S;
    if (i != j) qb[e] = x.value(b, m, upper_index(i, j, S)) * pb[j];
  }
  for (int i = threadIdx.x >> 5; i < S; i += blockDim.x >> 5) {
    const double s = row_sum(S, [&](int j) {
      return __dmul_rn(j == i ? 0.0 : x.value(b, m, upper_index(i, j, S)), pb[j]);  // (0 of a NaN or infinity is NaN)
    });
    if ((threadIdx.x & 31) == 0) qb[i * S + i] = __dsub_rn(__dmul_rn(0.0, pb[i]), s);
  }
}

// dL/dr_ij = (G_ij - G_ii) pi_j + (G_ji - G_jj) pi_i, dL/dpi_j = sum_i (G_ij - G_ii) r_ij
template <typename Map>
__global__ void __launch_bounds__(256) exch_q_backward_kernel(const __grid_constant__ Exch<Map> x, const double *pi, const double *G, int S,
                                                              double *d0, double *d1, double *d2, double *dpi) {
  __shared__ double red[3][8];
  __shared__ uint32_t sm[Exch<Map>::kMapped ? PairMap::kWords : 1];
  const int8_t *m = x.stage(sm);
  const int b = blockIdx.x, tid = threadIdx.x;
  const double *pb = pi + size_t(b) * S, *g = G + size_t(b) * S * S;
  double acc[3] = {0.0, 0.0, 0.0};
  for (int e = tid; e < S * S; e += 256) {
    const int i = e / S, j = e - i * S;
    if (i >= j) continue;
    const double d = (g[e] - g[i * S + i]) * pb[j] + (g[j * S + i] - g[j * S + j]) * pb[i];
    const int u = upper_index(i, j, S);
    if constexpr (!Exch<Map>::kMapped) {
      if (d0) d0[size_t(b) * x.count + u] = d;
    } else {
      const int m0 = m[u], m1 = m[x.count + u];
      const double v0 = x.param(b, m0), v1 = x.param(b, m1);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (m0 == c) acc[c] = fma(d, v1, acc[c]);
        if (m1 == c) acc[c] = fma(d, v0, acc[c]);
      }
    }
  }
  if (dpi)
    for (int j = tid; j < S; j += 256) {
      double s = 0.0;
      for (int i = 0; i < S; ++i)
        if (i != j) s = fma(g[i * S + j] - g[i * S + i], x.value(b, m, upper_index(i, j, S)), s);
      dpi[size_t(b) * S + j] = s;
    }
  if (!Exch<Map>::kMapped) return;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double s = lane_sum(acc[c]);
    if ((tid & 31) == 0) red[c][tid >> 5] = s;
  }
  __syncthreads();
  if (tid < 3) {  // one parameter per array
    double s = 0.0;
    for (int w = 0; w < 8; ++w) s += red[tid][w];
    double *d = tid == 0 ? d0 : (tid == 1 ? d1 : d2);
    if (d) d[b] = s;
  }
}

// ------------------------------------------------------- whole evaluations
// What one evaluation leaves for its gradient (doubles, per plan): normalised
// Q, mu, node lengths, rates, category weights, frequencies, eigen system.
struct Work {
  double *qn, *mu, *bl, *rates, *props, *pi, *lam, *u, *w;
  static size_t count(const tt_plan *p) {
    const size_t b = p->batch, S = p->S;
    return b * (3 * S * S + 2 * S + p->B + 2 * size_t(p->K) + 1);
  }
  Work(const tt_plan *p, double *base) {
    const size_t b = p->batch, S = p->S;
    double *x = base;
    auto take = [&](size_t n) {
      double *r = x;
      x += n;
      return r;
    };
    qn = take(b * S * S), u = take(b * S * S), w = take(b * S * S);
    lam = take(b * S), pi = take(b * S);
    bl = take(b * p->B), rates = take(b * p->K), props = take(b * p->K), mu = take(b);
  }
};

// mu = -sum_i pi_i Q_ii, Q / mu; node lengths (a zero after the free ones), and
// the category weights (row stride ps) as contiguous rows
__global__ void __launch_bounds__(256) prepare_kernel(const double *q, const double *pi, const double *bl, int nbl,
                                                      const double *rates, const double *props, long long ps, int S,
                                                      int B, int K, Work w) {
  __shared__ double smu;
  const int b = blockIdx.x, tid = threadIdx.x;
  const double *qb = q + size_t(b) * S * S, *pb = pi + size_t(b) * S;
  if (tid < 32) {
    const double s = -row_sum(S, [&](int i) { return __dmul_rn(qb[i * S + i], pb[i]); });
    if (tid == 0) smu = s, w.mu[b] = s;
  }
  __syncthreads();
  const double mu = smu;
  for (int e = tid; e < S * S; e += 256) w.qn[size_t(b) * S * S + e] = qb[e] / mu;
  for (int e = tid; e < B; e += 256) w.bl[size_t(b) * B + e] = e < nbl ? bl[size_t(b) * nbl + e] : 0.0;
  for (int e = tid; e < S; e += 256) w.pi[size_t(b) * S + e] = pb[e];
  for (int e = tid; e < K; e += 256) {
    w.rates[size_t(b) * K + e] = rates[size_t(b) * K + e];
    w.props[size_t(b) * K + e] = props[b * ps + e];
  }
}

// Chain from dlnL/dQ of the normalised matrix (d) to Q and the frequencies, all
// gradients times the sample's incoming gradient: with s = sum_ij d_ij Qn_ij,
//   dQ_ij = (d_ij + [i = j] pi_i s) / mu,  dpi_i = dpi_root_i + s Qn_ii.
__global__ void __launch_bounds__(256) finish_kernel(Work w, const double *d, const double *dt, const double *dr,
                                                     const double *dc, const double *dpi_root, const double *grad,
                                                     long long gs, int S, int B, int K, int nbl, double *dq,
                                                     double *dpi, double *dbl, double *drates, double *dprops) {
  __shared__ double red[8];
  const int b = blockIdx.x, tid = threadIdx.x;
  const double *qn = w.qn + size_t(b) * S * S, *db = d + size_t(b) * S * S;
  double s = 0.0;
  for (int e = tid; e < S * S; e += 256) s = fma(db[e], qn[e], s);
  s = lane_sum(s);
  if ((tid & 31) == 0) red[tid >> 5] = s;
  __syncthreads();
  s = 0.0;
#pragma unroll
  for (int i = 0; i < 8; ++i) s += red[i];
  const double g = grad[b * gs], mu = w.mu[b];
  if (dq)
    for (int e = tid; e < S * S; e += 256) {
      const int i = e / S;
      dq[size_t(b) * S * S + e] = g * ((e == i * S + i ? fma(w.pi[size_t(b) * S + i], s, db[e]) : db[e]) / mu);
    }
  if (dpi)
    for (int i = tid; i < S; i += 256)
      dpi[size_t(b) * S + i] = g * fma(s, qn[i * S + i], dpi_root[size_t(b) * S + i]);
  if (dbl)
    for (int e = tid; e < nbl; e += 256) dbl[size_t(b) * nbl + e] = g * dt[size_t(b) * B + e];
  for (int e = tid; e < K; e += 256) {
    if (drates) drates[size_t(b) * K + e] = g * dr[size_t(b) * K + e];
    if (dprops) dprops[size_t(b) * K + e] = g * dc[size_t(b) * K + e];
  }
}

template <typename Map>
Exch<Map> exch_of(int32_t S, const int32_t *counts, const double *p0, const double *p1, const double *p2,
                  const int8_t *map) {
  Exch<Map> x;
  x.p[0] = p0, x.p[1] = p1, x.p[2] = p2;
  for (int i = 0; i < 3; ++i) x.n[i] = counts[i];
  x.count = S * (S - 1) / 2;
  if constexpr (Exch<Map>::kMapped) std::memcpy(x.map.m, map, 2 * size_t(x.count));
  return x;
}

// the argument rules of the two rate-matrix calls
// (a map's entries lie in [-1, 2] and name parameters that exist)
int exch_check(int32_t batch, int32_t S, const int32_t *counts, const double *p0, const double *p1, const double *p2,
               const int8_t *map, const double *pi) {
  if (!counts || !p0 || !pi || batch < 1 || S < 2 || S > 64) return sfail(TT_ERR_INVALID_ARGUMENT, "rate matrix: NULL argument, empty batch or state count outside [2, 64]");
  const double *p[3] = {p0, p1, p2};
  for (int i = 0; i < 3; ++i) {
    if ((counts[i] > 0) != (p[i] != nullptr) || counts[i] < 0) return sfail(TT_ERR_INVALID_ARGUMENT, "rate matrix: parameter counts and pointers differ");
    if (map && counts[i] > 1) return sfail(TT_ERR_INVALID_ARGUMENT, "rate matrix: mapped parameters are scalars");
  }
  if (map)
    for (int e = 0; e < S * (S - 1); ++e)
      if (map[e] < -1 || map[e] >= counts[0] + counts[1] + counts[2])
        return sfail(TT_ERR_INVALID_ARGUMENT, "rate matrix: the map names a parameter that is not given");
  if (!map && (counts[0] != S * (S - 1) / 2 || counts[1] || counts[2]))
    return sfail(TT_ERR_INVALID_ARGUMENT, "rate matrix: expected S (S - 1) / 2 exchangeabilities");
  return TT_OK;
}

}  // namespace
}  // namespace tt

extern "C" {

int tt_weibull_rates(int32_t batch, int32_t category_count, const double *shape, double *rates, double *drates_dshape,
                     double *weights, void *stream) {
  using namespace tt;
  if (!shape || !rates || !drates_dshape || !weights || batch < 1 || category_count < 1 || category_count > 32)
    return sfail(TT_ERR_INVALID_ARGUMENT, "category rates: NULL argument, empty batch or more than 32 categories");
  weibull_rates_kernel<<<batch, 32, 0, static_cast<cudaStream_t>(stream)>>>(shape, category_count, rates,
                                                                            drates_dshape, weights);
  return sdone(cudaGetLastError(), "Weibull rates launch");
}

int tt_gamma_rates(int32_t batch, int32_t category_count, const double *shape, double *rates, double *drates_dshape,
                   double *weights, void *stream) {
  using namespace tt;
  if (!shape || !rates || !drates_dshape || !weights || batch < 1 || category_count < 1 || category_count > 32)
    return sfail(TT_ERR_INVALID_ARGUMENT, "category rates: NULL argument, empty batch or more than 32 categories");
  gamma_rates_kernel<<<batch, 32 * std::min(category_count, 8), 0, static_cast<cudaStream_t>(stream)>>>(
      shape, category_count, rates, drates_dshape, weights);
  return sdone(cudaGetLastError(), "Gamma rates launch");
}

int tt_rates_backward(int32_t batch, int32_t category_count, const double *grad_rates, const double *drates_dshape,
                      double *grad_shape, void *stream) {
  using namespace tt;
  if (!grad_rates || !drates_dshape || !grad_shape || batch < 1 || category_count < 1 || category_count > 32)
    return sfail(TT_ERR_INVALID_ARGUMENT, "category rates: NULL argument, empty batch or more than 32 categories");
  rates_backward_kernel<<<batch, 32, 0, static_cast<cudaStream_t>(stream)>>>(grad_rates, drates_dshape,
                                                                             category_count, grad_shape);
  return sdone(cudaGetLastError(), "category rates backward launch");
}

int tt_exchangeability_q(int32_t batch, int32_t state_count, const int32_t *param_counts, const double *params0,
                         const double *params1, const double *params2, const int8_t *map, const double *frequencies,
                         double *q, void *stream) {
  using namespace tt;
  const int rc = exch_check(batch, state_count, param_counts, params0, params1, params2, map, frequencies);
  if (rc) return rc;
  if (!q) return sfail(TT_ERR_INVALID_ARGUMENT, "NULL argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (map)
    exch_q_kernel<<<batch, 256, 0, s>>>(
        exch_of<PairMap>(state_count, param_counts, params0, params1, params2, map), frequencies, state_count, q);
  else
    exch_q_kernel<<<batch, 256, 0, s>>>(
        exch_of<NoMap>(state_count, param_counts, params0, params1, params2, map), frequencies, state_count, q);
  return sdone(cudaGetLastError(), "rate matrix launch");
}

int tt_exchangeability_q_backward(int32_t batch, int32_t state_count, const int32_t *param_counts,
                                  const double *params0, const double *params1, const double *params2,
                                  const int8_t *map, const double *frequencies, const double *grad_q,
                                  double *grad_params0, double *grad_params1, double *grad_params2,
                                  double *grad_frequencies, void *stream) {
  using namespace tt;
  const int rc = exch_check(batch, state_count, param_counts, params0, params1, params2, map, frequencies);
  if (rc) return rc;
  if (!grad_q) return sfail(TT_ERR_INVALID_ARGUMENT, "NULL argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (map)
    exch_q_backward_kernel<<<batch, 256, 0, s>>>(
        exch_of<PairMap>(state_count, param_counts, params0, params1, params2, map), frequencies, grad_q, state_count,
        grad_params0, grad_params1, grad_params2, grad_frequencies);
  else
    exch_q_backward_kernel<<<batch, 256, 0, s>>>(
        exch_of<NoMap>(state_count, param_counts, params0, params1, params2, map), frequencies, grad_q, state_count,
        grad_params0, grad_params1, grad_params2, grad_frequencies);
  return sdone(cudaGetLastError(), "rate matrix backward launch");
}

int tt_evaluate_workspace(const tt_plan *p, int64_t *work, int64_t *scratch) {
  using namespace tt;
  if (!p || !work || !scratch) return sfail(TT_ERR_INVALID_ARGUMENT, "NULL argument");
  *work = int64_t(Work::count(p));
  *scratch = int64_t(p->batch) * (int64_t(p->S) * p->S + p->B + p->K);
  return TT_OK;
}

int tt_evaluate(tt_plan *p, const double *q, const double *frequencies, const double *branch_lengths,
                int32_t lengths_per_sample, const double *rates, const double *category_weights,
                int64_t weights_stride, int32_t rescale, int32_t keep_partials, double *work,
                double *log_likelihood, void *stream) {
  using namespace tt;
  if (!p || !q || !frequencies || !branch_lengths || !rates || !category_weights || !work || !log_likelihood)
    return sfail(TT_ERR_INVALID_ARGUMENT, "NULL argument");
  if (lengths_per_sample < 1 || lengths_per_sample > p->B)
    return sfail(TT_ERR_INVALID_ARGUMENT, "tt_evaluate takes at most 2T-2 lengths per sample");
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return sdone(e, "cudaGetDevice");
  if (dev != p->device)  // before the first launch
    return sfail(TT_ERR_INVALID_ARGUMENT, "the current CUDA device differs from the plan's device");
  const Work w(p, work);
  prepare_kernel<<<p->batch, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      q, frequencies, branch_lengths, lengths_per_sample, rates, category_weights, weights_stride, p->S, p->B, p->K, w);
  int rc = sdone(cudaGetLastError(), "evaluation set-up launch");
  if (!rc) rc = tt_reversible_eigen(p->batch, p->S, w.qn, w.pi, w.lam, w.u, w.w, p->d_status, stream);
  if (!rc) rc = tt_update_transition_matrices(p, w.lam, w.u, w.w, w.bl, w.rates, stream);
  if (!rc) rc = tt_log_likelihood(p, w.props, w.pi, rescale, keep_partials, log_likelihood, nullptr, stream);
  return rc;
}

int tt_evaluate_gradient(tt_plan *p, double *work, const double *grad_log_likelihood, int64_t grad_stride,
                         int32_t lengths_per_sample, double *scratch, double *grad_q, double *grad_frequencies,
                         double *grad_branch_lengths, double *grad_rates, double *grad_weights, void *stream) {
  using namespace tt;
  if (!p || !work || !grad_log_likelihood || !scratch) return sfail(TT_ERR_INVALID_ARGUMENT, "NULL argument");
  if (lengths_per_sample < 1 || lengths_per_sample > p->B)
    return sfail(TT_ERR_INVALID_ARGUMENT, "tt_evaluate takes at most 2T-2 lengths per sample");
  const Work w(p, work);
  const size_t b = p->batch, S = p->S;
  double *d = scratch, *dt = d + b * S * S, *dr = dt + b * p->B;
  int rc = tt_gradient(p, w.props, w.pi, nullptr, nullptr, nullptr, stream);
  if (!rc) rc = tt_rate_matrix_gradient(p, w.lam, w.u, w.w, w.bl, w.rates, d, dt, dr, stream);
  if (rc) return rc;
  finish_kernel<<<p->batch, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      w, d, dt, dr, p->d_rootgrad + b * S, p->d_rootgrad, grad_log_likelihood, grad_stride, p->S, p->B, p->K, lengths_per_sample, grad_q,
      grad_frequencies, grad_branch_lengths, grad_rates, grad_weights);
  return sdone(cudaGetLastError(), "gradient finish launch");
}

}  // extern "C"
