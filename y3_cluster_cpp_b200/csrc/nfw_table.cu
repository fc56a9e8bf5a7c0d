// nfw_table.cu -- coefficients of the DeltaSigma polynomials (nfw_table.cuh).
#include <cmath>
#include <vector>

#include "nfw_table.cuh"

namespace y3b {

namespace {

// DeltaSigma(sqrt(w)) in extended precision, the branches of
// NfwUnit<double>: near w = 1 the series g = sum v^n / (2n + 1),
// Sigma = sum v^n / (2n + 3), v = 1 - w; below x = 1/2 the form of Sigma_bar
// without cancelling terms.
long double
dsigma_ld(long double w)
{
  const long double x = sqrtl(w), v = 1.0L - w;
  if (fabsl(v) < 0.25L) {
    long double g = 0.0L, s = 0.0L;
    for (int n = 34; n >= 0; --n) {
      g = 1.0L / (2 * n + 1) + v * g;
      s = 1.0L / (2 * n + 3) + v * s;
    }
    return 2.0L * (g + logl(0.5L * x)) / w - s;
  }
  if (x > 1.0L) {
    const long double y = sqrtl(-v), g = atanl(y) / y;
    return 2.0L * (g + logl(0.5L * x)) / w - (g - 1.0L) / v;
  }
  const long double y = sqrtl(v), g = logl((1.0L + y) / x) / y;
  if (x < 0.5L) {
    const long double bar =
      (2.0L / y) * (logl(2.0L / x) / (1.0L + y) + log1pl(-w / (2.0L * (1.0L + y))) / w);
    return bar - (g - 1.0L) / v;
  }
  return 2.0L * (g + logl(0.5L * x)) / w - (g - 1.0L) / v;
}

std::vector<double>
build()
{
  constexpr int N = kNfwCoef;
  const long double pi = 3.14159265358979323846264338327950288L;
  std::vector<double> out((size_t)kNfwSegs * N);
  // Chebyshev polynomials as monomials: T[k][j], y^j of T_k(y).
  long double T[N][N] = {};
  T[0][0] = 1.0L;
  T[1][1] = 1.0L;
  for (int k = 2; k < N; ++k)
    for (int j = 0; j < N; ++j) T[k][j] = (j ? 2.0L * T[k - 1][j - 1] : 0.0L) - T[k - 2][j];
  long double cs[N][N];  // cs[k][i] = T_k at the Chebyshev node i
  for (int k = 0; k < N; ++k)
    for (int i = 0; i < N; ++i) cs[k][i] = cosl(pi * k * (i + 0.5L) / N);
  const long double half = ldexpl(1.0L, -kNfwBits - 1);  // half a segment, in the mantissa
  for (int s = 0; s < kNfwSegs; ++s) {
    const int e = kNfwE0 + (s >> kNfwBits), b = s & ((1 << kNfwBits) - 1);
    const long double centre = 1.0L + (2 * b + 1) * half;
    long double f[N], mono[N] = {};
    for (int i = 0; i < N; ++i)
      f[i] = dsigma_ld(ldexpl(centre + half * cs[1][i], e));
    for (int k = 0; k < N; ++k) {
      long double c = 0.0L;
      for (int i = 0; i < N; ++i) c += f[i] * cs[k][i];
      c *= (k ? 2.0L : 1.0L) / N;
      for (int j = 0; j < N; ++j) mono[j] += c * T[k][j];
    }
    long double scale = 1.0L;
    for (int j = 0; j < N; ++j, scale /= half)
      out[((size_t)(j / 2) * kNfwSegs + s) * 2 + j % 2] = (double)(mono[j] * scale);
  }
  return out;
}

}  // namespace

const double*
nfw_table_host()
{
  static const std::vector<double> table = build();
  return table.data();
}

}  // namespace y3b
