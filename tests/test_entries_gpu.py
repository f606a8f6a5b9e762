"""Direct J/K over contraction lengths around the entry size of the pair lists
(1, 7, 8, 9 and 17 primitives per shell, so pairs of 1 to 289 primitives and up
to 37 entries), for every angular class, against the oracle.

Tolerance: an element sums n^2 <= 324 products of size <= 10, each in up to
37 x 37 parts, in another order than the oracle: 324 * 10 * 1.1e-16 = 4e-13 for
the sum, as much again for the parts; 2e-12 leaves a factor two.
"""
import numpy as np
import pytest

import oracle
from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet
from molecular2_b200.engine import IntegralEngine

pytestmark = pytest.mark.gpu
TOL = 2e-12


def contracted(l, n, atom, lo, hi):
    exps = np.geomspace(hi, lo, n) if n > 1 else np.array([lo])
    return (l, [float(x) for x in exps], [float(0.3 + 0.1 * k) for k in range(n)], atom)


def basis(lens, spherical=True):
    mol = geometry.water()
    shells = [contracted(l, n, k % 3, 0.15 + 0.1 * l, 40.0 / (1 + l)) for k, (l, n) in enumerate(lens)]
    return BasisSet.from_shells(shells, mol, spherical=spherical)


CASES = [
    [(0, 17), (0, 8), (0, 9), (0, 7), (0, 1)],
    [(0, 9), (1, 9), (1, 8), (0, 1), (1, 1)],
    [(2, 3), (1, 7), (2, 1), (0, 8), (1, 2)],
]


@pytest.mark.parametrize("lens", CASES)
@pytest.mark.parametrize("spherical", [True, False])
def test_direct_contraction_lengths(lens, spherical):
    obs = basis(lens, spherical)
    rng = np.random.default_rng(3)
    Da, Db = ((lambda c: c @ c.T)(rng.normal(size=(obs.nbf, 3)) * 0.3) for _ in range(2))
    Q = oracle.schwarz(obs)
    eng = IntegralEngine(obs)
    J, K = eng.jk_direct(Da, 1e-14)
    Jr, Kr, nq = oracle.jk_direct(obs, Da, Q, 1e-14)
    assert eng.last_quartets() == nq
    assert max(np.abs(J - Jr).max(), np.abs(K - Kr).max()) < TOL
    *refs, nq = oracle.jk_direct_uhf(obs, Da, Db, Q, 1e-14)
    for got, ref in zip(eng.jk_direct_uhf(Da, Db, 1e-14), refs):
        assert np.abs(got - ref).max() < TOL
