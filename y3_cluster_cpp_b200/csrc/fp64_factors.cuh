// fp64_factors.cuh -- the factors of exp(-(l - mu)^2 / 2 s^2) = F G H of the
// FP64 form (fp64_form.cu), mu = alpha + beta, with centred delta = l - L0,
// a = alpha - A0, b = beta - B0:
//   F = exp(-(delta - a)^2 c), G = exp(2 delta b c), H = exp(-b (2 a + b) c),
//   c = 1 / 2 s^2.
// Their exponents reach hundreds where s is small or mu far away while the
// product's is moderate, so an exponent's rounding must not scale with it:
// differences and products carry their rounding errors (Knuth's two-sum,
// products by fma), and exp(hi + lo) = exp(hi) (1 + lo).  Each factor is then
// good to about two units in the last place whatever its exponent; plain
// FP64 exponents cost 1e-14 of a cell at s = 0.06 and 5e-14 at 0.04.
// Plain functions, compiled for the device and (for the test of that bound)
// for the host.
#pragma once

#include <cmath>

#ifndef Y3B_HD
#ifdef __CUDACC__
#define Y3B_HD __host__ __device__ __forceinline__
#else
#define Y3B_HD inline
#endif
#endif

namespace y3b {

struct Dd {  // hi + lo, |lo| at most half a unit of hi
  double hi, lo;
};

Y3B_HD Dd
dd_diff(double x, double y)
{
  const double s = x - y, v = s - x;
  return {s, (x - (s - v)) - (y + v)};
}

Y3B_HD Dd
dd_mul(Dd x, Dd y)
{
  const double p = x.hi * y.hi;
  return {p, fma(x.hi, y.hi, -p) + fma(x.hi, y.lo, x.lo * y.hi)};
}

Y3B_HD double
dd_exp(Dd x)
{
  const double e = exp(x.hi);
  return fma(e, x.lo, e);
}

Y3B_HD Dd
f64_half_inv_var(double s)  // 1 / 2 s^2
{
  const double v = s * s, c = 0.5 / v;
  return {c, (fma(-c, v, 0.5) - c * fma(s, s, -v)) / v};
}

Y3B_HD double
f64_F(Dd delta, Dd a, Dd c)
{
  Dd d = dd_diff(delta.hi, a.hi);
  d.lo += delta.lo - a.lo;
  const Dd q = dd_mul(dd_mul(d, d), c);
  return dd_exp({-q.hi, -q.lo});
}

Y3B_HD double
f64_G(Dd delta, Dd b, Dd c)
{
  const Dd q = dd_mul(dd_mul(delta, b), c);
  return dd_exp({2.0 * q.hi, 2.0 * q.lo});
}

// H / exp(ln_d)
Y3B_HD double
f64_H(Dd a, Dd b, Dd c, double ln_d)
{
  Dd s = dd_diff(2.0 * a.hi, -b.hi);
  s.lo += 2.0 * a.lo + b.lo;
  const Dd q = dd_mul(dd_mul(b, s), c);
  const Dd x = dd_diff(-q.hi, ln_d);
  return dd_exp({x.hi, x.lo - q.lo});
}

}  // namespace y3b
