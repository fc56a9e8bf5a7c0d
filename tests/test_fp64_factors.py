"""The factors of the FP64 form's Gaussian (csrc/fp64_factors.cuh), compiled
for the host, against 60-digit values.  u = 2^-53 below."""
import ctypes as C
import os
import subprocess

import mpmath as mp
import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "y3_cluster_cpp_b200", "csrc")
U = 2.0 ** -53
SRC = """
#include "fp64_factors.cuh"
using namespace y3b;
extern "C" void factors(double l, double al, double be, double A0, double B0, double s, double* o)
{
  const Dd d = dd_diff(l, A0 + B0), a = dd_diff(al, A0), b = dd_diff(be, B0);
  const Dd c = f64_half_inv_var(s);
  o[0] = f64_F(d, a, c);
  o[1] = f64_G(d, b, c);
  o[2] = f64_H(a, b, c, 0.0);
  o[3] = f64_H(a, b, c, 0.5 * b.hi * b.hi * c.hi);
}
"""


@pytest.fixture(scope="module")
def factors(tmp_path_factory):
    d = tmp_path_factory.mktemp("fp64_factors")
    src, so = d / "f.cpp", d / "f.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC,
                    str(src), "-o", str(so)], check=True)
    fn = C.CDLL(str(so)).factors
    fn.argtypes = [C.c_double] * 6 + [C.POINTER(C.c_double)]
    return fn


@pytest.mark.parametrize("s", [0.02, 0.04, 0.1, 0.2, 1.0])
def test_factors(factors, s):
    """Each factor to 4 u (the exponential's one and a half, the correction's
    two roundings), with exponents up to 700 and nodes near zero; the
    factorised Gaussian to the factors' sum."""
    rng = np.random.default_rng(7)
    out = (C.c_double * 4)()
    worst = 0
    with mp.workdps(60):
        for n in range(600):
            A0, B0 = np.rint(rng.uniform(-2, 5, 2) * 2 ** 20) / 2 ** 20
            l = rng.uniform(0, 7) if n % 3 else 10 ** rng.uniform(-5, 0)
            al = A0 + rng.normal() * 10 * s
            be = B0 + rng.uniform(-0.4, 0.4) * min(1.0, 10 * s)
            if n % 2:  # near the Gaussian's peak
                al = l - be + rng.normal() * 4 * s
            factors(l, al, be, A0, B0, s, out)
            L, AL, BE, a0, b0, S = map(mp.mpf, map(float, (l, al, be, A0, B0, s)))
            c = 1 / (2 * S * S)
            d, a, b = L - a0 - b0, AL - a0, BE - b0
            ln_d = mp.mpf(0.5 * float(be - B0) * float(be - B0) * (0.5 / (s * s)))
            e = [-(d - a) ** 2 * c, 2 * d * b * c, -b * (2 * a + b) * c]
            for got, x in zip(out, e + [e[2] - ln_d]):
                if abs(x) > 700:
                    continue
                # the fourth's ln_d is formed again here, to two units of it
                tol = 4 * U if got != out[3] else 4 * U + 4 * U * float(ln_d)
                assert abs(mp.mpf(got) / mp.exp(x) - 1) < tol, (l, al, be, x)
            if max(map(abs, e)) < 700:
                want = mp.exp(-(L - AL - BE) ** 2 * c)
                err = float(abs(mp.mpf(out[0]) * out[1] * out[2] / want - 1))
                worst = max(worst, err)
    assert worst < 12 * U
