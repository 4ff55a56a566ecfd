"""The fp64 3x3 solve and the reciprocal of the vertex update (warpvbd_b200/csrc/vbd_solve.h),
compiled for the host, against exact rational arithmetic: blocks of well-shaped tets, of
nearly incompressible ones (one stiff direction, lambda / mu up to 1e12) and of very different
scales."""
import ctypes
import os
import subprocess
from fractions import Fraction

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "warpvbd_b200",
                    "csrc")


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    d = tmp_path_factory.mktemp("solve3")
    src, so = d / "solve3.cpp", d / "solve3.so"
    src.write_text('#include "vbd_solve.h"\n'
                   'extern "C" int solve(const double* h, const double* g, double* x) {\n'
                   '  return vbd::solve3(h, g, x);\n}\n'
                   'extern "C" double newton(double x, double y) {\n'
                   '  return vbd::newton_reciprocal(x, y);\n}\n')
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-fPIC", "-shared",
                    f"-I{CSRC}", str(src), "-o", str(so)], check=True)
    return ctypes.CDLL(str(so))


@pytest.fixture(scope="module")
def solve3(library):
    f = library.solve
    f.argtypes = [ctypes.POINTER(ctypes.c_double)] * 3

    def run(h, g):
        h, g, x = np.array(h, float), np.array(g, float), np.zeros(3)
        p = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for a in (h, g, x)]
        return bool(f(*p)), x
    return run


def _exact(h, g):
    """-H^-1 g in rational arithmetic, by cofactors."""
    a = [Fraction(float(v)) for v in h]
    b = [Fraction(float(v)) for v in g]
    H = [[a[0], a[1], a[2]], [a[1], a[3], a[4]], [a[2], a[4], a[5]]]

    def cof(i, j):
        r, c = [k for k in range(3) if k != i], [k for k in range(3) if k != j]
        m = H[r[0]][c[0]] * H[r[1]][c[1]] - H[r[0]][c[1]] * H[r[1]][c[0]]
        return m if (i + j) % 2 == 0 else -m
    det = sum(H[0][j] * cof(0, j) for j in range(3))
    x = [-sum(cof(j, i) * b[j] for j in range(3)) / det for i in range(3)]
    minors = (a[0], a[0] * a[3] - a[1] * a[1], det)
    return x, all(m > 0 for m in minors)


def _packed(H):
    return H[np.triu_indices(3)]


@pytest.mark.parametrize("scale", [1.0, 1e-63, 1e-62, 1e62, 1e63, 1e-100, 1e100])
@pytest.mark.parametrize("k", [0.0, 1.0, 1e3, 1e5, 1e7, 1e9, 1e12])
def test_error_grows_with_the_condition_number_only(solve3, k, scale):
    """A backward-stable factorisation of a 3x3 positive definite matrix solves H + dH with
    |dH| <= (3n + 1) u |L| |D| |L^T| (Higham, Accuracy and Stability of Numerical Algorithms,
    10.1): a relative error of at most 3 (3n + 1) u cond(H) = 30 u cond(H) in the norm.  The
    elimination step with Cramer's rule on what is left keeps within it; from scales of
    1e-62 and 1e62 on its products leave the range and L D L^T is taken."""
    rng = np.random.default_rng(int(np.log10(k + 1)))
    for _ in range(60):
        c, M, g = rng.standard_normal(3), rng.standard_normal((3, 3)), rng.standard_normal(3)
        H = (M @ M.T + np.eye(3) + k * np.outer(c, c)) * scale
        ok, x = solve3(_packed(H), g)
        ref, spd = _exact(_packed(H), g)
        assert ok == spd
        if not spd:
            continue
        err = np.sqrt(sum(float((Fraction(float(v)) - r) * Fraction(scale)) ** 2
                          for v, r in zip(x, ref)))
        size = np.sqrt(sum(float(r * Fraction(scale)) ** 2 for r in ref))
        assert err <= 30 * 2.0 ** -53 * np.linalg.cond(H / scale) * size


@pytest.mark.parametrize("H", [
    np.diag([-1.0, 2.0, 3.0]), np.diag([1.0, -2.0, 3.0]), np.diag([1.0, 2.0, -3.0]),
    np.diag([0.0, 0.0, 0.0]), np.diag([1.0, 0.0, 1.0]),
    np.array([[1.0, 2.0, 0.0], [2.0, 1.0, 0.0], [0.0, 0.0, 1.0]]),
    np.full((3, 3), np.nan), np.diag([1.0, np.nan, 1.0]), -np.eye(3)])
def test_blocks_that_are_not_positive_definite_are_reported(solve3, H):
    assert not solve3(_packed(H), np.ones(3))[0]


@pytest.mark.parametrize("start", [-2.0 ** -20, -2.0 ** -24, 0.0, 2.0 ** -27, 2.0 ** -20])
def test_newton_reciprocal_is_rounded_once(library, start):
    """From an approximation with relative error e <= 2^-20 the first step leaves e^2 = 2^-40
    and two roundings, the second (2^-40 + 2^-52)^2 and one rounding of a term of that size:
    half a unit in the last place of the result, plus less than 2^-79 of it."""
    f = library.newton
    f.argtypes, f.restype = [ctypes.c_double, ctypes.c_double], ctypes.c_double
    rng = np.random.default_rng(7)
    for x in np.concatenate([1.0 + rng.random(400), 4.0 + rng.random(400) * 1e-6,
                             10.0 ** rng.uniform(0, 300, 400)]):
        y = f(x, (1.0 / x) * (1.0 + start))
        exact = 1 / Fraction(float(x))
        assert abs(Fraction(y) - exact) <= (Fraction(float(np.spacing(y))) / 2
                                            + exact / 2 ** 79)
