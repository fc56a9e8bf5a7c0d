// mor_norm.cuh -- the normalisation of the lognormal MOR on the lam_t domain.
#pragma once

#include "common.cuh"

namespace y3b {

// MOR normalisation D = Phi(b) - Phi(a) in FP64, a = (l_lo - mu)/s,
// b = (l_hi - mu)/s.  The lam_t domain is many sigma wide, so at most one
// tail is open: D = 1 exactly when both are below half an FP64 ulp
// (a < -8.5, b > 8.5); with one tail closed D = Phi(b) or Phi(-a), a single
// erfc on the side that does not cancel.  Kept out of line: the rare path.
static __device__ __noinline__ double
mor_norm_slow(double a, double b)
{
  constexpr double kInvSqrt2 = 0.70710678118654752440;
  if (a < -8.5)  // low tail closed: D = Phi(b)
    return b < 0.0 ? 0.5 * erfc(-b * kInvSqrt2) : 1.0 - 0.5 * erfc(b * kInvSqrt2);
  if (b > 8.5)  // high tail closed: D = Phi(-a)
    return a > 0.0 ? 0.5 * erfc(a * kInvSqrt2) : 1.0 - 0.5 * erfc(-a * kInvSqrt2);
  return phi_diff(a, b);
}

__device__ __forceinline__ double
mor_norm(double a, double b)
{
  if (a < -8.5 && b > 8.5) return 1.0;
  return mor_norm_slow(a, b);
}

// ln D for the same D, finite where D itself underflows FP64 (mu more than
// ~38 sigma outside the lam_t domain).  With Q(x) = erfc(x / sqrt 2) / 2 =
// erfcx(x / sqrt 2) exp(-x^2 / 2) / 2: for 0 < a < b, D = Q(a) - Q(b) and
// ln D = ln Q(a) + log1p(-Q(b) / Q(a)); for a < b < 0, D = Q(-b) - Q(-a)
// likewise; otherwise mu lies inside the domain and D is not small.
static __device__ __noinline__ double
ln_mor_norm(double a, double b)
{
  constexpr double kInvSqrt2 = 0.70710678118654752440;
  if (a > 0.0) {
    const double ra = erfcx(a * kInvSqrt2), rb = erfcx(b * kInvSqrt2);
    return log(0.5 * ra) - 0.5 * a * a + log1p(-(rb / ra) * exp(-0.5 * (b - a) * (b + a)));
  }
  if (b < 0.0) {
    const double ra = erfcx(-a * kInvSqrt2), rb = erfcx(-b * kInvSqrt2);
    return log(0.5 * rb) - 0.5 * b * b + log1p(-(ra / rb) * exp(-0.5 * (a - b) * (a + b)));
  }
  return log(mor_norm(a, b));
}

}  // namespace y3b
