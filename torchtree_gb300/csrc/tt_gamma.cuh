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

// digamma for a > 0
TT_HD inline double digamma_pos(double a) {
  double acc = 0.0;
  while (a < 10.0) {
    acc -= 1.0 / a;
    a += 1.0;
  }
  const double r = 1.0 / a, r2 = r * r;
  // ln a - 1/(2a) - sum_k B_2k / (2k a^2k), k = 1..6
  const double series =
      r2 * (1.0 / 12.0 - r2 * (1.0 / 120.0 - r2 * (1.0 / 252.0 - r2 * (1.0 / 240.0 - r2 * (1.0 / 132.0 -
                                                                                          r2 * (691.0 / 32760.0))))));
  return acc + log(a) - 0.5 * r - series;
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

// The iteration ends with a step below this share of x: Halley's method is of
// third order, so the error left after such a step is rounding alone.  (A bound
// at rounding itself, 4e-16, is met by chance only: the steps then wander by an
// ulp or two until the iteration limit.)
constexpr double kGammaStep = 1e-13;

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

// Halley's step from x to xn, from p = P(a, x) and scale = x^a e^-x / Gamma(a);
// false when the density is not usable
TT_HD inline bool gamma_halley(double a, double q, double x, double p, double scale, double &xn) {
  const double dfdx = scale / x;  // x^(a-1) e^-x / Gamma(a)
  if (!(dfdx > 0.0) || !isfinite(dfdx)) return false;
  const double u = (p - q) / dfdx;
  xn = x - u / (1.0 - 0.5 * fmin(1.0, u * ((a - 1.0) / x - 1.0)));
  if (xn <= 0.0) xn = 0.5 * x;
  return true;
}

// x with P(a, x) = q and dx/da; false for invalid input or no convergence
TT_HD inline bool gamma_quantile(double a, double q, double &x_out, double &dxda_out) {
  if (!(a > 0.0) || !(q > 0.0) || !(q < 1.0) || !isfinite(a)) return false;
  const double lga = lgamma(a);
  double x = gamma_start(a, q);
  double p = 0.0, z = 0.0, scale = 0.0, delta = 0.0;
  for (int it = 0; it < 100; ++it) {
    if (!(x > 0.0)) x = 1e-300;
    if (!gamma_p_series(a, x, lga, p, z, scale)) return false;
    double xn;
    if (!gamma_halley(a, q, x, p, scale, xn)) return false;
    delta = fabs(xn - x);
    x = xn;
    if (delta <= kGammaStep * x) break;
  }
  if (!(delta <= kGammaStep * x)) return false;
  if (!gamma_p_series(a, x, lga, p, z, scale)) return false;
  x_out = x;
  dxda_out = -x * (p * (log(x) - digamma_pos(a)) - z) / scale;
  return true;
}

#ifdef __CUDACC__
// The device form: one warp per quantile, every lane with the same a, q and x.
// The serial series is a chain of two FP64 divisions and two multiplications
// per term (2.0 ms for any batch that fits the GPU: the chain, not the
// throughput, bounds it).  Here lane j holds term 32 c + j + 1 of chunk c: one
// division per lane, the running product T_n and the harmonic sum H_n by warp
// scans, the sums by butterflies (every lane ends with the same bits).  Most
// quantiles of a site model need one chunk.  4 quantiles 1,094 -> 35 us, 256
// quantiles 2,101 -> 37 us.
__device__ inline bool gamma_p_series_warp(double a, double x, double lga, bool want_z, double &p, double &z,
                                           double &scale) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  scale = exp(gamma_log_scale(a, x, lga));
  double term = scale / a, h = 1.0 / a;  // of the last term added
  p = term;
  z = term * h;
  for (int n0 = 1; n0 < 200000; n0 += 32) {
    const double d = a + double(n0 + lane);
    double prod = x / d, sum = want_z ? 1.0 / d : 0.0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double y = __shfl_up_sync(kAll, prod, o);
      const double g = want_z ? __shfl_up_sync(kAll, sum, o) : 0.0;
      if (lane >= o) {
        prod *= y;
        if (want_z) sum += g;
      }
    }
    const double tn = term * prod, hn = h + sum;
    double ps = tn, zs = want_z ? tn * hn : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ps += __shfl_xor_sync(kAll, ps, o);
      if (want_z) zs += __shfl_xor_sync(kAll, zs, o);
    }
    p += ps;
    z += zs;
    term = __shfl_sync(kAll, tn, 31);
    h = __shfl_sync(kAll, hn, 31);
    if (term <= p * 1e-17 && (!want_z || term * h <= z * 1e-17)) return true;
  }
  return false;
}

// digamma for a > 0 by a warp: the recurrence's terms across the lanes
__device__ inline double digamma_pos_warp(double a) {
  const int m = a < 10.0 ? int(ceil(10.0 - a)) : 0, lane = threadIdx.x & 31;
  double acc = lane < m ? 1.0 / (a + lane) : 0.0;
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);  // m <= 10: lanes 0-15
  acc = __shfl_sync(0xffffffffu, acc, 0);
  return digamma_pos(a + m) - acc;
}

// The quantile to about 1e-6 in FP32, by the same iteration: an FP64 step of it takes
// about 3 us (64 cycles per instruction and SM quarter), an FP32 one a tenth of that.
// 0 where FP32 does not serve: shapes outside [0.05, 20] (underflow, cancellation in
// the scale) or no convergence.  Rates of one sample: 44 -> 26 us.
__device__ inline float gamma_quantile_f32_warp(float a, float q, float lga, float x) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  if (!(a >= 0.05f && a <= 20.0f && x > 1e-30f && x < 1e30f)) return 0.0f;
  for (int it = 0; it < 12; ++it) {
    const float scale = expf(a * logf(x) - x - lga);
    float term = scale / a, p = term;
    for (int n0 = 1; n0 < 512 && term > p * 1e-8f; n0 += 32) {
      float prod = x / (a + float(n0 + lane));
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const float y = __shfl_up_sync(kAll, prod, o);
        if (lane >= o) prod *= y;
      }
      const float tn = term * prod;
      float ps = tn;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) ps += __shfl_xor_sync(kAll, ps, o);
      p += ps;
      term = __shfl_sync(kAll, tn, 31);
    }
    const float dfdx = scale / x;
    if (!(dfdx > 1e-30f) || !isfinite(dfdx)) return 0.0f;
    const float u = (p - q) / dfdx;
    float xn = x - u / (1.0f - 0.5f * fminf(1.0f, u * ((a - 1.0f) / x - 1.0f)));
    if (xn <= 0.0f) xn = 0.5f * x;
    const float delta = fabsf(xn - x);
    x = xn;
    if (!(x > 1e-30f) || !isfinite(x)) return 0.0f;
    if (delta <= 1e-5f * x) return x;
  }
  return 0.0f;
}

// gamma_quantile by a warp; the same result in every lane
__device__ inline bool gamma_quantile_warp(double a, double q, double &x_out, double &dxda_out) {
  if (!(a > 0.0) || !(q > 0.0) || !(q < 1.0) || !isfinite(a)) return false;
  const double lga = lgamma(a);
  double x = gamma_start(a, q), p = 0.0, z = 0.0, scale = 0.0, delta = 0.0;
  const float x32 = gamma_quantile_f32_warp(float(a), float(q), float(lga), float(x));
  if (x32 > 0.0f) x = double(x32);
  for (int it = 0; it < 100; ++it) {
    if (!(x > 0.0)) x = 1e-300;
    if (!gamma_p_series_warp(a, x, lga, false, p, z, scale)) return false;
    double xn;
    if (!gamma_halley(a, q, x, p, scale, xn)) return false;
    delta = fabs(xn - x);
    x = xn;
    // an error of 1e-6 before the step is one of about 1e-18 after it (third order)
    if (delta <= (x32 > 0.0f ? 1e-6 : kGammaStep) * x) break;
  }
  if (!(delta <= (x32 > 0.0f ? 1e-6 : kGammaStep) * x)) return false;
  if (!gamma_p_series_warp(a, x, lga, true, p, z, scale)) return false;
  x_out = x;
  dxda_out = -x * (p * (log(x) - digamma_pos_warp(a)) - z) / scale;
  return true;
}
#endif

}  // namespace tt
