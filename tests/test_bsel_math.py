"""The arctangent, two-disk overlap and shifted-Poisson density of the
selection-bias kernels (csrc/bsel_math.cuh), compiled for the host, against
50-digit values.  u = 2^-53 below."""
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
#include "bsel_math.cuh"
extern "C" {
double atan01(double q) { return y3b::atan01(q); }
double lens_area(double t, double o, double l) { return y3b::lens_area(t, o, l); }
double shifted_poisson(double x, double lam) { return y3b::shifted_poisson(x, lam); }
}
"""


@pytest.fixture(scope="module")
def fn(tmp_path_factory):
    d = tmp_path_factory.mktemp("bsel_math")
    src, so = d / "m.cpp", d / "m.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC,
                    str(src), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    for name, n in (("atan01", 1), ("lens_area", 3), ("shifted_poisson", 2)):
        getattr(lib, name).restype = C.c_double
        getattr(lib, name).argtypes = [C.c_double] * n
    return lib


def test_no_reciprocal_root_by_hand():
    """Square roots and their reciprocals come from CUDA's own functions: no
    approximate FP64 instruction is refined in this source."""
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh", ".h", ".cpp")):
            text = open(os.path.join(CSRC, f)).read()
            for op in ("rsqrt.approx", "rcp.approx", "sqrt.approx"):
                assert op not in text, (f, op)


def test_atan01(fn):
    """Truncation 3e-17 and the roundings of z q (two), the Horner sum and the
    last addition: below 2 u relative (the sum is at most 0.22 q)."""
    q = np.concatenate([np.linspace(0.0, 1.0, 2001), np.geomspace(1e-300, 1.0, 300)])
    with mp.workdps(50):
        for v in q[q > 0]:
            want = mp.atan(mp.mpf(float(v)))
            assert abs(mp.mpf(fn.atan01(float(v))) / want - 1) < 2 * U, v
    assert fn.atan01(0.0) == 0.0


def test_lens_area(fn):
    """Against the textbook area of the lens, in 50 digits: the two sectors and
    the triangles are each good to ~10 u of the smaller disk's scale."""
    rng = np.random.default_rng(5)
    with mp.workdps(50):
        for _ in range(400):
            o, l = np.exp(rng.uniform(-9, -3, 2))
            f = rng.choice([rng.uniform(), 10 ** rng.uniform(-12, -3),
                            1 - 10 ** rng.uniform(-12, -3)])
            t = abs(o - l) + f * (o + l - abs(o - l))
            if not abs(o - l) < t <= o + l:
                continue
            T, O, L = mp.mpf(t), mp.mpf(o), mp.mpf(l)
            c1 = (T * T + L * L - O * O) / (2 * T * L)
            c2 = (T * T + O * O - L * L) / (2 * T * O)
            sq = max((-T + L + O) * (T + L - O) * (T - L + O) * (T + L + O), 0)
            clip = lambda c: min(max(c, -1), 1)
            want = L * L * mp.acos(clip(c1)) + O * O * mp.acos(clip(c2)) - mp.sqrt(sq) / 2
            # s1..s4 carry a rounding of the radii: near tangency a half angle,
            # the root of a small side, moves by the root of it, weighted by
            # the opposite small side's own area: scale of the triangle.
            tol = 10 * U * float(O * O + L * L)
            assert abs(fn.lens_area(t, o, l) - float(want)) < tol, (t, o, l)


def _poisson(x, lam):
    x, lam = mp.mpf(x), mp.mpf(lam)
    return mp.exp(-lam + (x - 1) * mp.log(lam) - mp.loggamma(x))


def test_shifted_poisson(fn):
    """Relative error: a few roundings, plus those of the exponent's terms,
    (x - 1) times the logarithm (absolute error 4 u from its argument, and
    half a unit of its own), y - lam, and their sum."""
    rng = np.random.default_rng(6)
    xs = np.concatenate([10 ** rng.uniform(-6, 3, 1500), [1e-6, 1.0, 2.0, 1000.0]])
    ls = np.concatenate([10 ** rng.uniform(-3, 3, 1500), [1e-300, 1e-300, 1e3, 1e3]])
    near = rng.uniform(size=1500) < 0.6   # most weight lies near the peak
    xs[:1500][near] = np.maximum(1e-6, ls[:1500][near] * (1 + rng.normal(size=near.sum()) * 0.2))
    rel = []
    with mp.workdps(60):
        for x, lam in zip(map(float, xs), map(float, ls)):
            want = _poisson(x, lam)
            if want < mp.mpf("1e-290"):
                continue
            err = float(abs(mp.mpf(fn.shifted_poisson(x, lam)) / want - 1))
            ln = abs(np.log(lam / (x + 10)))
            tol = U * (40 + abs(x - 1) * (5 + 2 * ln) + 3 * abs(x + 10 - lam))
            assert err < tol, (x, lam, err, tol)
            if lam <= 1e3 and lam > 1e-3:
                rel.append(err)
    rms = float(np.sqrt(np.mean(np.square(rel))))
    assert len(rel) > 500 and rms < 1.5e-13, rms   # 7e-14 over x and lam up to 1e3
