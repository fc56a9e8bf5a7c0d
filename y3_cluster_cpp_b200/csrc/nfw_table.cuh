// nfw_table.cuh -- the projected NFW excess DeltaSigma(x) = Sigma_bar - Sigma
// (unit of 2 r_s delta_c rho) as a piecewise polynomial in w = x^2.
//
// The miscentred profiles evaluate DeltaSigma at millions of offsets: the
// closed form costs an artanh or arctan, a log, square roots and divisions
// in FP64 (~250 instructions with divergent branches), the polynomial two
// integer operations, one subtraction and eight multiply-adds.  DeltaSigma
// is analytic in w away from w = 0, so on a segment [a, a (1 + 1/32)] the
// degree-7 Chebyshev interpolant converges as 130^-8 ~ 1e-17: the segment is
// the exponent and the top five mantissa bits of w, the variable the
// distance of the mantissa from the segment's centre.  Coefficients are
// formed on the host in extended precision from the closed form.  Outside
// [2^-36, 2^22) (x from 4e-6 to 2000) the closed form itself is evaluated.
#pragma once

#include "common.cuh"
#include "host_common.h"

namespace y3b {

constexpr int kNfwBits = 5;                                // segments per octave: 32
constexpr int kNfwE0 = -36, kNfwE1 = 22;                   // w in [2^kNfwE0, 2^kNfwE1)
constexpr int kNfwSegs = (kNfwE1 - kNfwE0) << kNfwBits;    // 1856
constexpr int kNfwCoef = 8;                                // 64 bytes a segment, 116 KB

// Coefficient pairs [kNfwCoef / 2][kNfwSegs][2], formed once per process:
// lanes whose w lie on neighbouring segments read neighbouring 16-byte words.
const double* nfw_table_host();

// DeltaSigma(sqrt(w)); tab in global memory (16-byte aligned).  A w outside
// the range (NaN too) sets `outside`, and the caller evaluates the
// closed form instead: no call in the inner loops, whose registers would be
// spilled around it.
__device__ __forceinline__ double
nfw_dsigma_w(const double* __restrict__ tab, double w, bool& outside)
{
  const int hi = __double2hiint(w);
  const int s = (hi >> (20 - kNfwBits)) - ((1023 + kNfwE0) << kNfwBits);
  outside |= (unsigned)s >= (unsigned)kNfwSegs;
  const int seg = min((unsigned)s, (unsigned)(kNfwSegs - 1));
  const double m = __hiloint2double((hi & 0xFFFFF) | 0x3FF00000, __double2loint(w));
  const int keep = ((1 << kNfwBits) - 1) << (20 - kNfwBits);
  const double t =
    m - __hiloint2double((hi & keep) | 0x3FF00000 | (1 << (19 - kNfwBits)), 0);
  const double2* c = reinterpret_cast<const double2*>(tab) + seg;
  const double2 c0 = __ldg(c), c1 = __ldg(c + kNfwSegs), c2 = __ldg(c + 2 * kNfwSegs),
                c3 = __ldg(c + 3 * kNfwSegs);
  const double t2 = t * t;
  const double lo = fma(fma(c1.y, t, c1.x), t2, fma(c0.y, t, c0.x));
  const double up = fma(fma(c3.y, t, c3.x), t2, fma(c2.y, t, c2.x));
  return fma(up, t2 * t2, lo);
}

}  // namespace y3b
