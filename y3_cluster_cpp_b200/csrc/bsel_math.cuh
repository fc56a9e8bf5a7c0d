// bsel_math.cuh -- the two-disk overlap and the shifted-Poisson density of the
// selection-bias operators.  Plain FP64 functions, compiled for the device and
// (for the tests of their bounds) for the host.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define Y3B_HD __host__ __device__ __forceinline__
#else
#define Y3B_HD inline
#endif

namespace y3b {

constexpr double kBselPi = 3.14159265358979323846;
constexpr double kInvSqrt2Pi = 0.39894228040143267794;  // 1 / sqrt(2 pi)

Y3B_HD double
inv_sqrt(double v)
{
#ifdef __CUDA_ARCH__
  return rsqrt(v);
#else
  return 1.0 / std::sqrt(v);
#endif
}

// atan on [0, 1]: atan(q) / q as a degree-19 polynomial in q^2 (Chebyshev
// interpolation of the function, truncation 3e-17).
Y3B_HD double
atan01(double q)
{
  const double z = q * q;
  double s = -1.93423475928923002e-05;
  s = fma(s, z, 2.14238107386039464e-04);
  s = fma(s, z, -1.12525443022346450e-03);
  s = fma(s, z, 3.75113848396514118e-03);
  s = fma(s, z, -8.99108054265826059e-03);
  s = fma(s, z, 1.67195960635073901e-02);
  s = fma(s, z, -2.55686236443717387e-02);
  s = fma(s, z, 3.38712670270067476e-02);
  s = fma(s, z, -4.08112475031788546e-02);
  s = fma(s, z, 4.66874530484852890e-02);
  s = fma(s, z, -5.23742347191881660e-02);
  s = fma(s, z, 5.87682811448727235e-02);
  s = fma(s, z, -6.66576491068972266e-02);
  s = fma(s, z, 7.69219899745829383e-02);
  s = fma(s, z, -9.09089979321734132e-02);
  s = fma(s, z, 1.11111105780020827e-01);
  s = fma(s, z, -1.42857142669267329e-01);
  s = fma(s, z, 1.99999999996479605e-01);
  s = fma(s, z, -3.33333333333307003e-01);
  return fma(s, z * q, q);
}

// Overlap area of two disks of radii o and l at distance t, partially
// overlapping, |o - l| < t <= o + l (p_op_detail::area_overlap,
// p_operator_cuhre_t.hh:97-125), from the triangle with sides t, l, o: with
// s1 = o + l - t, s2 = t - (o - l), s3 = t + (o - l), s4 = t + l + o and
// y = sqrt(s1 s2 s3 s4) (four times its area), the half angles at the two
// centres have the tangents s1 s3 / y and s1 s2 / y, reciprocals s2 s4 / y and
// s3 s4 / y.  One reciprocal square root and two polynomials in place of two
// acos, three divisions and a square root, and no digits are lost near
// tangency.
Y3B_HD double
lens_area(double t, double o, double l)
{
  const double d = o - l, s1 = (o + l) - t, s2 = t - d, s3 = t + d, s4 = (o + l) + t;
  const double a = s1 * s3, b = s2 * s4, c = s1 * s2, e = s3 * s4;
  const double sq = fmax(a * b, 1e-290), r = inv_sqrt(sq);
  const bool big1 = a > b, big2 = c > e;  // tangent above 1: the complement of the angle
  const double h1 = atan01((big1 ? b : a) * r), h2 = atan01((big2 ? e : c) * r);
  const double a1 = big1 ? 0.5 * kBselPi - h1 : h1, a2 = big2 ? 0.5 * kBselPi - h2 : h2;
  return fma(2.0 * (l * l), a1, fma(2.0 * (o * o), a2, -0.5 * (sq * r)));
}

// Shifted-Poisson density exp(-lam + (x - 1) ln lam) / Gamma(x).  With
// y = x + 10, 1 / Gamma(x) = prod_{i<10} (x + i) / Gamma(y) and Stirling's
// series for Gamma(y) (seven terms, remainder below 3e-17), grouped so that
// the exponent (x - 1) ln(lam / y) + y - lam is free of large cancelling
// terms: relative error 7e-14 rms over x and lam up to 1e3, 9e-13 for
// exp(-lam + (x - 1) ln lam - lgamma(x)), at a third of the instructions.
Y3B_HD double
shifted_poisson(double x, double lam)
{
  const double y = x + 10.0, q = inv_sqrt(y), r = q * q, r2 = r * r, r4 = r2 * r2;
  double s = fma(r2, 1.0 / 156.0, -691.0 / 360360.0);
  s = fma(s, r2, 1.0 / 1188.0);
  s = fma(s, r2, -1.0 / 1680.0);
  s = fma(s, r2, 1.0 / 1260.0);
  s = fma(s, r2, -1.0 / 360.0);
  s = fma(s, r2, 1.0 / 12.0);
  const double p = (x * (x + 1.0)) * ((x + 2.0) * (x + 3.0)) * ((x + 4.0) * (x + 5.0)) *
                   ((x + 6.0) * (x + 7.0)) * ((x + 8.0) * (x + 9.0)) * (r4 * r4 * r2);
  return kInvSqrt2Pi * p * q * exp((x - 1.0) * log(lam * r) + ((y - lam) - s * r));
}

}  // namespace y3b
