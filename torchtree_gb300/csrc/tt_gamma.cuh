// Quantiles of the Gamma(shape a, rate 1) distribution and their derivative
// with respect to the shape, in FP64, on the host and the device.
//
// The discretised Gamma site model takes the category rates at the
// quantiles (2k+1)/(2K), divided by their mean (the same construction as
// torchtree's discretised Weibull model, site_model.py:173-195).  With the
// Gamma(a, rate a) distribution the quantile is x/a, where x solves
// P(a, x) = q for the regularised lower incomplete gamma function
//
//   P(a, x) = gamma(a, x) / Gamma(a),
//   gamma(a, x) = x^a e^-x S0,   S0 = sum_n x^n / (a (a+1) ... (a+n))
//
// (the power series of Abramowitz & Stegun 6.5.29; every term is positive).
// The root is found by Halley's method on f(x) = P(a, x) - q with
// f'(x) = x^(a-1) e^-x / Gamma(a) and f''/f' = (a-1)/x - 1, from the
// starting points of Numerical Recipes (Press et al., 3rd ed., section 6.2.1:
// Abramowitz & Stegun 26.2.23 with the Wilson-Hilferty transform for a > 1,
// the small-x power law for a <= 1).
//
// The shape derivative is analytic.  Differentiating the series term by term,
// d S0 / da = -S1 with S1 = sum_n T_n H_n, T_n = x^n / (a (a+1) ... (a+n))
// and H_n = sum_(j<=n) 1/(a+j), so
//
//   dP/da = x^a e^-x / Gamma(a) * (S0 (ln x - psi(a)) - S1),
//   dx/da = -(dP/da) / (dP/dx) = -x (S0 (ln x - psi(a)) - S1),
//
// with psi the digamma function (recurrence psi(a) = psi(a+1) - 1/a up to
// a >= 10, then the asymptotic series of Abramowitz & Stegun 6.3.18).
#pragma once

#include <math.h>

namespace tt {

#ifdef __CUDACC__
#define TT_HD __host__ __device__
#else
#define TT_HD
#endif

// acc + digamma of a >= 10
TT_HD inline double digamma_tail(double a, double acc) {
  const double r = 1.0 / a, r2 = r * r;
  // ln a - 1/(2a) - sum_k B_2k / (2k a^2k), k = 1..6
  const double series =
      r2 * (1.0 / 12.0 - r2 * (1.0 / 120.0 - r2 * (1.0 / 252.0 - r2 * (1.0 / 240.0 - r2 * (1.0 / 132.0 -
                                                                                          r2 * (691.0 / 32760.0))))));
  return acc + log(a) - 0.5 * r - series;
}

// digamma for a > 0
TT_HD inline double digamma_pos(double a) {
  double acc = 0.0;
  while (a < 10.0) {
    acc -= 1.0 / a;
    a += 1.0;
  }
  return digamma_tail(a, acc);
}

// log(x^a e^-x / Gamma(a)).  For a >= 10 the large terms a ln x, x and
// ln Gamma(a) nearly cancel; with x = a (1 + t) and Stirling's series for
// ln Gamma (Abramowitz & Stegun 6.1.41) it is
//   ln(a / 2 pi) / 2 - c(a) + a (ln(1 + t) - t),
// c(a) = 1/(12a) - 1/(360a^3) + 1/(1260a^5) - 1/(1680a^7) + 1/(1188a^9) - ...
TT_HD inline double gamma_log_scale(double a, double x, double lga) {
  if (a < 10.0) return a * log(x) - x - lga;
  const double r = 1.0 / a, r2 = r * r;
  const double c = r * (1.0 / 12.0 - r2 * (1.0 / 360.0 - r2 * (1.0 / 1260.0 - r2 * (1.0 / 1680.0 -
                                                                                 r2 * (1.0 / 1188.0)))));
  const double t = (x - a) / a;
  return 0.5 * log(a / 6.283185307179586) - c + a * (log1p(t) - t);
}

// The series at (a, x), scaled to P: p = P(a, x) = sum_n p_n with
// p_n = scale T_n, z = sum_n p_n H_n = scale S1, and scale = x^a e^-x / Gamma(a)
// (the terms stay below 1, so nothing overflows for large a and x).
// False if the series did not converge.
TT_HD inline bool gamma_p_series(double a, double x, double lga, double &p, double &z, double &scale) {
  scale = exp(gamma_log_scale(a, x, lga));
  double term = scale / a, h = 1.0 / a;
  p = term;
  z = term * h;
  for (int n = 1; n < 200000; ++n) {
    term *= x / (a + n);
    h += 1.0 / (a + n);
    p += term;
    z += term * h;
    if (term <= p * 1e-17 && term * h <= z * 1e-17) return true;
  }
  return false;
}

// The iteration ends with a step below kGammaStop of x, at most kGammaSteps steps, and
// counts as converged when the last one is below kGammaStep.  Rounding leaves steps of
// an ulp or two, so which of the neighbouring values the iteration ends with depends on
// every rounding on its way.
constexpr int kGammaSteps = 100;
constexpr double kGammaStop = 4e-16, kGammaStep = 1e-13;

// the starting point of the iteration (Numerical Recipes 6.2.1)
TT_HD inline double gamma_start(double a, double q) {
  double x;
  if (a > 1.0) {
    const double pp = q < 0.5 ? q : 1.0 - q;
    const double t = sqrt(-2.0 * log(pp));
    double zq = (2.30753 + t * 0.27061) / (1.0 + t * (0.99229 + t * 0.04481)) - t;
    if (q < 0.5) zq = -zq;
    const double w = 1.0 - 1.0 / (9.0 * a) - zq / (3.0 * sqrt(a));
    x = fmax(1e-3, a * w * w * w);
  } else {
    const double t = 1.0 - a * (0.253 + a * 0.12);
    x = q < t ? pow(q / t, 1.0 / a) : 1.0 - log(1.0 - (q - t) / (1.0 - t));
  }
  return x;
}

// Halley's step from x to xn, from p = P(a, x), the density x^(a-1) e^-x / Gamma(a) and
// curve = (a - 1) / x; false when the density is not usable
TT_HD inline bool gamma_step(double q, double x, double p, double density, double curve, double &xn) {
  if (!(density > 0.0) || !isfinite(density)) return false;
  const double u = (p - q) / density;
  xn = x - u / (1.0 - 0.5 * fmin(1.0, u * (curve - 1.0)));
  if (xn <= 0.0) xn = 0.5 * x;
  return true;
}

// x with P(a, x) = q and dx/da; false for invalid input or no convergence
TT_HD inline bool gamma_quantile(double a, double q, double &x_out, double &dxda_out) {
  if (!(a > 0.0) || !(q > 0.0) || !(q < 1.0) || !isfinite(a)) return false;
  const double lga = lgamma(a);
  double x = gamma_start(a, q);
  double p = 0.0, z = 0.0, scale = 0.0, delta = 0.0;
  for (int it = 0; it < kGammaSteps; ++it) {
    if (!(x > 0.0)) x = 1e-300;
    if (!gamma_p_series(a, x, lga, p, z, scale)) return false;
    double xn;
    if (!gamma_step(q, x, p, scale / x, (a - 1.0) / x, xn)) return false;
    delta = fabs(xn - x);
    x = xn;
    if (delta <= kGammaStop * x) break;
  }
  if (!(delta <= kGammaStep * x)) return false;
  if (!gamma_p_series(a, x, lga, p, z, scale)) return false;
  x_out = x;
  dxda_out = -x * (p * (log(x) - digamma_pos(a)) - z) / scale;
  return true;
}

#ifdef __CUDACC__
// The device form: one warp per quantile, every lane with the same a, q and x, and
// gamma_quantile's value to the last bit: FP32 transition matrices are rounded from
// the category rates, and rates that move by 1e-16 take some of 1e8 entries to the
// neighbouring FP32 value and gradients by 1e-9 with them.  So every rounding of the
// serial form stays (its products and sums are not contracted), and the time goes out elsewhere:
//  * the divisions of 28 terms and three more run at once, one per lane (an FP64
//    division is nine instructions of 64 cycles, the chain of term and sum only two);
//  * the sums stop where a term can no longer round into them, on the integer pipe;
//  * an iteration that never comes below kGammaStop wanders through a few neighbouring
//    values, the next a function of the last: the lanes keep all values, and once one
//    comes back, where step kGammaSteps ends is known without taking the steps.
// Shapes around 0.5, 4 categories: 1 / 16 / 64 samples 49 / 82 / 95 us (the longest of
// their iterations).  One thread per quantile, every step taken: 1,094 us for 4
// quantiles, 2,101 for 256.
constexpr unsigned kGammaLanes = 0xffffffffu;
constexpr int kGammaChunk = 28;  // terms per round of divisions; lanes 28 - 30 hold three other quotients

__device__ __forceinline__ int gamma_exponent(double v) { return __double2hiint(v) >> 20; }  // biased; v >= 0

// gamma_p_series and, for gamma_step, density = scale / x and curve = (a - 1) / x
template <bool WANT_Z>
__device__ __forceinline__ bool gamma_p_series_warp(double a, double x, double lga, double &p, double &z,
                                                    double &scale, double &density, double &curve) {
  const int lane = threadIdx.x & 31;
  scale = exp(gamma_log_scale(a, x, lga));
  if (!isfinite(scale)) return false;
  double term = 0.0, h = 0.0;  // of the last term added
  for (int n0 = 1; n0 < 200000; n0 += kGammaChunk) {
    const double d = a + double(n0 + lane);
    const double num = lane < kGammaChunk ? x : lane == 30 ? a - 1.0 : scale;
    const double den = lane < kGammaChunk ? d : lane == 28 ? a : x;
    const double ratio = num / den;
    double inv = 0.0;
    if constexpr (WANT_Z) inv = 1.0 / (lane < kGammaChunk ? d : a);
    if (n0 == 1) {
      p = term = __shfl_sync(kGammaLanes, ratio, 28);
      density = __shfl_sync(kGammaLanes, ratio, 29);
      curve = __shfl_sync(kGammaLanes, ratio, 30);
      if constexpr (WANT_Z) {
        h = __shfl_sync(kGammaLanes, inv, 28);
        z = __dmul_rn(term, h);
      }
    }
#pragma unroll 1
    for (int j0 = 0; j0 < kGammaChunk; j0 += 4) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        term = __dmul_rn(term, __shfl_sync(kGammaLanes, ratio, j0 + j));
        p = __dadd_rn(p, term);
        if constexpr (WANT_Z) {
          h = __dadd_rn(h, __shfl_sync(kGammaLanes, inv, j0 + j));
          z = __dadd_rn(z, __dmul_rn(term, h));
        }
      }
      // a term below 2^-55 of the sum does not change it, nor do those after it
      const int ep = gamma_exponent(p), et = gamma_exponent(term);
      bool done = ep < 64 ? term <= p * 1e-17 : ep - et >= 56;  // (the exponents of tiny sums do not tell)
      if constexpr (WANT_Z) {
        const int ez = gamma_exponent(z), eh = gamma_exponent(h) - 1023;
        done = done && (ez < 64 ? term * h <= z * 1e-17 : ez - (et + eh + 1) >= 56);
      }
      if (done) return true;
    }
  }
  return false;
}

// digamma_pos by a warp: the recurrence's divisions across the lanes, its sum in order
__device__ inline double digamma_pos_warp(double a) {
  const int lane = threadIdx.x & 31;
  double mine = a, acc = 0.0;
  int m = 0;
  for (; a < 10.0; ++m) {  // at most 10
    if (lane == m) mine = a;
    a += 1.0;
  }
  const double inv = 1.0 / mine;
  for (int j = 0; j < m; ++j) acc -= __shfl_sync(kGammaLanes, inv, j);
  return digamma_tail(a, acc);
}

// gamma_quantile by a warp; the same result in every lane
__device__ inline bool gamma_quantile_warp(double a, double q, double &x_out, double &dxda_out) {
  if (!(a > 0.0) || !(q > 0.0) || !(q < 1.0) || !isfinite(a)) return false;
  const int lane = threadIdx.x & 31;
  const double lga = lgamma(a);
  double x = gamma_start(a, q), p = 0.0, z = 0.0, scale = 0.0, delta = 0.0, density = 0.0, curve = 0.0;
  double seen[4] = {0.0, 0.0, 0.0, 0.0};  // the value at step 32 s + lane
  static_assert(kGammaSteps <= 128, "four values per lane");
  auto value_at = [&](int i) {
    const int s = i >> 5;
    return __shfl_sync(kGammaLanes, s == 0 ? seen[0] : s == 1 ? seen[1] : s == 2 ? seen[2] : seen[3], i & 31);
  };
  for (int it = 0; it < kGammaSteps; ++it) {
    if (!(x > 0.0)) x = 1e-300;
    int back = -1;  // the step that had this value
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const unsigned hit = __ballot_sync(kGammaLanes, seen[s] == x);
      if (hit) back = 32 * s + __ffs(hit) - 1;
    }
    if (back >= 0) {  // no step of this cycle ends the iteration
      const int period = it - back;
      x = value_at(back + (kGammaSteps - back) % period);
      delta = fabs(x - value_at(back + (kGammaSteps - 1 - back) % period));
      break;
    }
#pragma unroll
    for (int s = 0; s < 4; ++s)
      if (it == 32 * s + lane) seen[s] = x;
    if (!gamma_p_series_warp<false>(a, x, lga, p, z, scale, density, curve)) return false;
    double xn;
    if (!gamma_step(q, x, p, density, curve, xn)) return false;
    delta = fabs(xn - x);
    x = xn;
    if (delta <= kGammaStop * x) break;
  }
  if (!(delta <= kGammaStep * x)) return false;
  if (!gamma_p_series_warp<true>(a, x, lga, p, z, scale, density, curve)) return false;
  x_out = x;
  dxda_out = -x * (p * (log(x) - digamma_pos_warp(a)) - z) / scale;
  return true;
}
#endif

}  // namespace tt
