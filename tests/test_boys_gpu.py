"""The Boys function of the integral kernels, every order as the top one, against
extended precision (64-bit mantissa).

Tolerances, in units u = 1.1e-16.  Below T = 36 + 3M the top order is a table
polynomial: its constant term, the last addition and a fifth of the one before
round, 2.7 u = 3e-16; each step down rounds a sum, a product and the constant it
multiplies with, 3 u = 3.4e-16.  Above, F_m is a constant times r^(2m+1), r = T^-1/2:
3.2 u for the constant, r and the product, 2 u for each factor 1/T.
"""
import numpy as np
import pytest

from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet
from molecular2_b200.engine import IntegralEngine

pytestmark = pytest.mark.gpu


def reference(T, M):
    """F_0 .. F_M: the series at M (positive terms), downward recursion."""
    assert np.finfo(np.longdouble).nmant >= 63
    T = T.astype(np.longdouble)
    F = np.zeros((M + 1, T.size), dtype=np.longdouble)
    term = np.full(T.size, 1.0, dtype=np.longdouble) / (2 * M + 1)
    F[M] = term
    for i in range(1, 2500):
        term = term * 2.0 * T / (2 * M + 2 * i + 1)
        F[M] += term
        if (term <= 1e-22 * F[M]).all():
            break
    e = np.exp(-T)
    F[M] *= e
    for m in range(M - 1, -1, -1):
        F[m] = (2.0 * T * F[m + 1] + e) / (2 * m + 1)
    return F


@pytest.fixture(scope="module")
def engine():
    return IntegralEngine(BasisSet(geometry.water(), "sto-3g"))


@pytest.mark.parametrize("M", range(10))
def test_boys(engine, M):
    rng = np.random.default_rng(M)
    top = 36.0 + 3.0 * M
    edges = 0.375 * np.arange(0, 180)
    T = np.concatenate([[0.0, 1e-300, 1e-20, 1e-12, top, np.nextafter(top, 0.0), np.nextafter(top, 99.0)],
                        edges, edges + 0.1875, np.nextafter(edges + 0.1875, 0.0), np.nextafter(edges + 0.1875, 99.0),
                        rng.uniform(0.0, 2.0, 4000), rng.uniform(0.0, 80.0, 20000), rng.uniform(80.0, 600.0, 1000),
                        10.0 ** rng.uniform(-10.0, 2.0, 2000)])
    got, ref = engine.boys_selftest(M, T), reference(T, M)
    err = np.abs((got - ref) / ref).astype(np.float64)
    m = np.arange(M + 1)[:, None]
    tol = np.where(T < top, 3e-16 + 3.4e-16 * (M - m), 3.6e-16 + 2.3e-16 * m)
    print(f"M {M}: below 36 + 3M top {err[M, T < top].max():.2e} all {err[:, T < top].max():.2e}, "
          f"above {err[:, T >= top].max():.2e}")
    assert (err <= tol).all()
