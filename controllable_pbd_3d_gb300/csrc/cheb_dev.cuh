// Device side of the Chebyshev interval: the largest eigenvalue of the Lanczos
// tridiagonal and the coefficients of the polynomial, by one warp.
#pragma once

#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>

#include "jform.cuh"

namespace mgpbd {
namespace jdev {

// Whether all k eigenvalues of the symmetric tridiagonal T (diagonal a,
// off-diagonal b) lie below x: the leading minors of T - x I alternate in sign,
// starting negative.  The minors by their three-term recurrence, T scaled by
// 1 / s (s bounds its eigenvalues, so the minors of 32 rows stay in range): no
// division, whose latency was most of the search's time.  (Eigenvalues that all
// lie within 1e-13 s of x, of 24 rows, or 3e-10 s, of 32, may make a minor 0: x
// then counts as not above them.)
__host__ __device__ inline bool all_below(const double* a, const double* b, int k, double x,
                                          double inv_s) {
  double p0 = 1.0, p1 = (a[0] - x) * inv_s;
  bool ok = p1 < 0.0;
  for (int i = 1; i < k; ++i) {
    const double c = b[i - 1] * inv_s;
    const double p = (a[i] - x) * inv_s * p1 - c * c * p0;
    p0 = p1;
    p1 = p;
    ok = ok && ((i & 1) ? p > 0.0 : p < 0.0);
  }
  return ok;
}

// Largest eigenvalue of T by Sturm multisection on its Gershgorin interval,
// one warp: each round the 32 lanes test 32 points that split the interval
// into 33 parts, and the interval shrinks to the part that holds the largest
// eigenvalue (the first point with all k below it is the new upper end),
// until its width is below 1e-12 of the upper end.  The result is the upper
// end, in all lanes.
__device__ inline double lanczos_lmax(const double* a, const double* b, int k) {
  const int lane = threadIdx.x & 31;
  double lo = 1e300, hi = -1e300, s = 0.0;
  for (int i = 0; i < k; ++i) {
    const double r = (i > 0 ? fabs(b[i - 1]) : 0.0) + (i + 1 < k ? fabs(b[i]) : 0.0);
    lo = fmin(lo, a[i] - r);
    hi = fmax(hi, a[i] + r);
  }
  s = fmax(fabs(lo), fabs(hi));
  if (!(hi >= lo) || !isfinite(hi) || !isfinite(lo)) return NAN;
  const double inv_s = s > 0.0 ? 1.0 / s : 1.0;
  for (int it = 0; it < 60 && hi - lo > __dmul_rn(1e-12, fmax(1.0, fabs(hi))); ++it) {
    const double step = (hi - lo) * (1.0 / 33.0);
    const double x = lane == 31 ? hi - step : lo + __dmul_rn(step, static_cast<double>(lane + 1));
    const unsigned all = __ballot_sync(0xffffffffu, all_below(a, b, k, x, inv_s));
    // the first point with every eigenvalue below it bounds the largest;
    // none: the largest lies above the last point
    const int f = all ? __ffs(all) - 1 : 32;
    const double nlo = f == 0 ? lo : __shfl_sync(0xffffffffu, x, f > 0 ? f - 1 : 0);
    const double nhi = f == 32 ? hi : __shfl_sync(0xffffffffu, x, f < 32 ? f : 31);
    lo = nlo;
    hi = nhi;
  }
  return hi;
}

// ... on the host, one point after the other
inline double host_lanczos_lmax(const double* a, const double* b, int k) {
  double lo = 1e300, hi = -1e300;
  for (int i = 0; i < k; ++i) {
    const double r = (i > 0 ? std::fabs(b[i - 1]) : 0.0) + (i + 1 < k ? std::fabs(b[i]) : 0.0);
    lo = std::fmin(lo, a[i] - r);
    hi = std::fmax(hi, a[i] + r);
  }
  const double s = std::fmax(std::fabs(lo), std::fabs(hi));
  if (!(hi >= lo) || !std::isfinite(hi) || !std::isfinite(lo)) return NAN;
  const double inv_s = s > 0.0 ? 1.0 / s : 1.0;
  for (int it = 0; it < 60 && hi - lo > 1e-12 * std::fmax(1.0, std::fabs(hi)); ++it) {
    const double step = (hi - lo) * (1.0 / 33.0);
    auto point = [&](int l) { return l == 31 ? hi - step : lo + step * (l + 1); };
    int f = 0;
    while (f < 32 && !all_below(a, b, k, point(f), inv_s)) ++f;
    const double nlo = f == 0 ? lo : point(f - 1), nhi = f == 32 ? hi : point(f);
    lo = nlo;
    hi = nhi;
  }
  return hi;
}

// Chebyshev acceleration coefficients on [hi * lo_ratio, hi], hi 2% above
// lmax (Saad, "Iterative Methods for Sparse Linear Systems", 2nd ed.,
// Alg. 12.1): sigma = theta / delta, rho_0 = 1 / sigma, rho_i = 1 / (2 sigma -
// rho_{i-1}), d_i = rho_i rho_{i-1} d_{i-1} + (2 rho_i / delta) r_i.  One
// thread; c1, c2 have kMaxCheb entries.  False when lmax is not finite and
// positive (the interval is then that of 2).
__device__ inline bool cheb_interval(double lmax, int degree, double lo_ratio, float* c1, float* c2,
                                     double* theta_out, float* inv_theta) {
  const bool ok = isfinite(lmax) && lmax > 0.0;
  const double hi = ok ? __dmul_rn(1.02, lmax) : 2.0;
  const double lo = __dmul_rn(hi, lo_ratio);
  const double theta = __dmul_rn(0.5, hi + lo), delta = __dmul_rn(0.5, hi - lo);
  const double sigma = __ddiv_rn(theta, delta);
  double rho = __ddiv_rn(1.0, sigma);
  for (int i = 0; i < kMaxCheb; ++i) c1[i] = c2[i] = 0.0f;
  for (int i = 1; i < degree && i < kMaxCheb; ++i) {
    const double rn = __ddiv_rn(1.0, __dmul_rn(2.0, sigma) - rho);
    c1[i] = static_cast<float>(__dmul_rn(rn, rho));
    c2[i] = static_cast<float>(__ddiv_rn(__dmul_rn(2.0, rn), delta));
    rho = rn;
  }
  *theta_out = theta;
  *inv_theta = static_cast<float>(__ddiv_rn(1.0, theta));
  return ok;
}

}  // namespace jdev
}  // namespace mgpbd
