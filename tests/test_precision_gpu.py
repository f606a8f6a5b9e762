"""The direct builds at thresholds of zero and far below the default keep the
integrals of pairs with tiny overlap: 200 s functions in a row, neighbours'
products of 4e-13, the density on the neighbours alone.

J of a pair of neighbours is then a sum of (pair|pair) integrals of 1e-25 and
less, known in closed form.  Its terms are products of about ten FP64 factors:
relative 1e-13.
"""
import math

import numpy as np
import pytest

from molecular2_b200.basis import BasisSet, Molecule
from molecular2_b200.engine import IntegralEngine

pytestmark = pytest.mark.gpu
N, STEP = 200, 7.6


def system():
    mol = Molecule(["h"] * N, [[0.0, 0.0, STEP * k] for k in range(N)], angstrom=False)
    obs = BasisSet.from_shells([(0, [1.0], [1.0], k) for k in range(N)], mol)
    D = np.zeros((N, N))
    i = np.arange(N - 1)
    D[i, i + 1] = D[i + 1, i] = 1.0
    norm = (2.0 / math.pi) ** 0.75
    z = mol.xyz[:, 2]  # 7.6 k is rounded, and e^{-R^2/2} sees it
    K = norm ** 2 * np.exp(-0.5 * (z[1:] - z[:-1]) ** 2)
    T = (0.5 * (z[1:] + z[:-1])[:, None] - 0.5 * (z[1:] + z[:-1])[None, :]) ** 2
    F0 = np.array([[0.5 * math.sqrt(math.pi / t) * math.erf(math.sqrt(t)) if t > 0 else 1.0 for t in row] for row in T])
    J = 2.0 * math.pi ** 2.5 / (2.0 * 2.0 * math.sqrt(4.0)) * 2.0 * K * (F0 @ K)
    return obs, D, J


@pytest.mark.parametrize("precision", [0.0, 1e-40])
def test_tiny_integrals_are_kept(precision):
    obs, D, ref = system()
    eng = IntegralEngine(obs)
    i = np.arange(N - 1)
    J, _ = eng.jk_direct(D, precision)
    assert np.abs(J[i, i + 1] / ref - 1.0).max() < 1e-13
    Ja, Jb, _, _ = eng.jk_direct_uhf(D, 0.5 * D, precision)
    assert np.abs(Ja[i, i + 1] / ref - 1.0).max() < 1e-13
    assert np.abs(Jb[i, i + 1] / ref - 0.5).max() < 1e-13
