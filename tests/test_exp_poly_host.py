"""The tensor exp's polynomials and plan (wannier90_gb300/csrc/k_oz_exp.cu), from the constants in the
source: T8 and T12 multiply out to the Taylor coefficients, the plan's norms bound the truncation, and
the scheme restated in NumPy -- plan from sqrt(||X^2||_1), polynomial, squarings, and the optimal step
from the trial step's powers -- agrees with the eigendecomposition."""
import math
import os
import re
from fractions import Fraction

import numpy as np
import pytest

SRC = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "wannier90_gb300", "csrc",
                        "k_oz_exp.cu")).read()
C = {n: Fraction(v) for n, v in re.findall(r"(kT\w+) = (-?[0-9.]+)", SRC)}
PLAN = [float(x) for x in re.findall(r"rho (?:<=|>) ([0-9.e-]+)f", SRC)]


def _mul(a, b):
    r = [Fraction(0)] * (len(a) + len(b) - 1)
    for i, x in enumerate(a):
        for j, y in enumerate(b):
            r[i + j] += x * y
    return r


def _add(*ps):
    return [sum((p[i] for p in ps if i < len(p)), Fraction(0)) for i in range(max(map(len, ps)))]


def _taylor(p, degree):
    assert len(p) == degree + 1
    for n, c in enumerate(p):
        assert abs(c * math.factorial(n) - 1) < Fraction(1, 10 ** 15), (n, float(c * math.factorial(n) - 1))


def test_t8_is_the_taylor_polynomial():
    x = {i: C["kT8x%d" % i] for i in range(1, 8)}
    A = _mul([0, 0, Fraction(1)], [0, x[1], x[2]])
    left = _add(A, [0, 0, x[3]])
    right = _add([x[4], x[5], x[6]], [x[7] * a for a in A])
    _taylor(_add(_mul(left, right), [1, 1, C["kT8y2"]]), 8)


def test_t12_is_the_taylor_polynomial():
    B4 = [0, C["kT12e1"], C["kT12e2"], C["kT12e3"]]
    A = _add(_mul(B4, B4), [0, 0, C["kT12a2"], C["kT12a3"]])
    B2 = [C["kT12b0"], C["kT12b1"], C["kT12b2"], C["kT12b3"]]
    _taylor(_add(_mul(_add(B2, A), A), [1, 1, C["kT12c2"], C["kT12c3"]]), 12)


def test_plan_bounds_the_truncation():
    t4, t8, t12 = PLAN
    for m, theta in ((4, t4), (8, t8), (12, t12)):
        # the tail of the series beyond its first term: theta / (m + 2) of it
        assert theta ** (m + 1) / math.factorial(m + 1) * (1 + theta / (m + 1)) <= 2.0 ** -53


def _plan(rho):
    t4, t8, t12 = PLAN
    if rho <= t4:
        return 4, 0
    if rho <= t8:
        return 8, 0
    js = 0
    while rho > t12 and js < 60:
        rho *= 0.5
        js += 1
    return 12, js


def _exp(X, P2, f, m, js):
    """exp(f 2^js ... ) of the kernel: coefficients carry f, the powers are X's own."""
    c = {k: float(v) for k, v in C.items()}
    W = len(X)
    eye = np.eye(W)
    f = f * 0.5 ** js
    if m == 4:
        E = P2 @ (f * f * (0.5 * eye + f / 6 * X + f * f / 24 * P2)) + eye + f * X
    elif m == 8:
        A = P2 @ (c["kT8x1"] * f ** 3 * X + c["kT8x2"] * f ** 4 * P2)
        E = ((A + c["kT8x3"] * f * f * P2) @ (c["kT8x4"] * eye + c["kT8x5"] * f * X + c["kT8x6"] * f * f * P2 + c["kT8x7"] * A)
             + eye + f * X + c["kT8y2"] * f * f * P2)
    else:
        P3 = P2 @ X
        B4 = c["kT12e1"] * f * X + c["kT12e2"] * f ** 2 * P2 + c["kT12e3"] * f ** 3 * P3
        A = B4 @ B4 + c["kT12a2"] * f ** 2 * P2 + c["kT12a3"] * f ** 3 * P3
        B2 = c["kT12b0"] * eye + c["kT12b1"] * f * X + c["kT12b2"] * f ** 2 * P2 + c["kT12b3"] * f ** 3 * P3
        E = (B2 + A) @ A + eye + f * X + c["kT12c2"] * f ** 2 * P2 + c["kT12c3"] * f ** 3 * P3
    for _ in range(js):
        E = E @ E
    return E


# norms on both sides of every step of the plan, W around its tile widths, and the optimal step at
# several multiples of the trial step
@pytest.mark.parametrize("W", [3, 8, 17, 32])
def test_scheme_against_the_eigendecomposition(W):
    rng = np.random.default_rng(W)
    for norm in [t * s for t in PLAN for s in (0.5, 0.999, 1.001, 1.9)] + [1e-12, 1.0, 5.0, 40.0]:
        X = rng.standard_normal((W, W)) + 1j * rng.standard_normal((W, W))
        X = X - X.conj().T
        X *= norm / np.linalg.norm(X, 2)
        P2 = X @ X
        rho = math.sqrt(np.abs(P2).sum(0).max())
        assert rho >= norm * (1 - 1e-12)
        w, V = np.linalg.eigh(1j * X)
        for f in (1.0, -0.3, 2.7, 100.0):
            m, js = _plan(rho * abs(f))
            got = _exp(X, P2, f, m, js)
            want = (V * np.exp(-1j * f * w)) @ V.conj().T
            # truncation 2^-53, W-term products, doubled by every squaring; the eigenvalues' own error
            tol = 2.0 ** -53 * (8 * W * 2 ** js + 8 * W * max(1.0, norm * abs(f)))
            assert np.abs(got - want).max() <= tol, (norm, f, m, js, np.abs(got - want).max(), tol)
