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


@pytest.mark.parametrize("lens", CASES)
def test_schwarz_and_one_body_contraction_lengths(lens):
    """Schwarz bounds (square roots of one integral, |Q| <= 2) and S, T, V (|V| <= 60; sums over up to 289
    primitives and 3 nuclei, 60 * 300 * 1.1e-16 = 2e-12; 5e-12 leaves a factor two)."""
    obs = basis(lens)
    eng = IntegralEngine(obs)
    assert np.abs(eng.getPrescreen() - oracle.schwarz(obs)).max() < 1e-13
    for got, ref in zip(eng.one_body(), oracle.one_body(obs)):
        assert np.abs(ref).max() < 60.0
        assert np.abs(got - ref).max() < 5e-12


@pytest.mark.parametrize("lens", CASES)
@pytest.mark.parametrize("spherical", [True, False])
def test_gradient_contraction_lengths(lens, spherical):
    """Terms are integrals times 2 alpha (alpha <= 40, |g| <= 100 a term), at most 324 x 289 of them:
    the sum's rounding is below 100 * sqrt(94,000) * 1.1e-16 = 3e-12; 2e-11 leaves a factor six."""
    obs = basis(lens, spherical)
    rng = np.random.default_rng(4)
    C = rng.normal(size=(obs.nbf, 3)) * 0.3
    D, W = 2.0 * C @ C.T, (C * np.array([-1.0, -0.7, -0.4])) @ C.T
    g, g2 = IntegralEngine(obs).compute_forces(D, W, 1e-14)
    ref2 = oracle.grad2e(obs, D, oracle.schwarz(obs), 1e-14)
    S1, T1, V1 = oracle.one_body_deriv(obs)
    na = obs.mol.natom
    ref = ref2 + obs.mol.enuc_grad() + np.array(
        [np.sum((T1[i] + V1[i]) * D) - 2.0 * np.sum(S1[i] * W) for i in range(3 * na)]).reshape(na, 3)
    assert max(np.abs(ref).max(), np.abs(ref2).max()) < 100.0
    assert max(np.abs(g - ref).max(), np.abs(g2 - ref2).max()) < 2e-11


@pytest.mark.parametrize("spherical", [True, False])
def test_one_body_is_symmetric_and_repeatable(spherical):
    """To the last bit, also for pairs of up to 37 entries and within a shell."""
    obs = basis([(0, 17), (1, 9), (2, 9), (0, 9), (2, 1)], spherical)
    eng = IntegralEngine(obs)
    ref = eng.one_body()
    for M in ref:
        assert np.array_equal(M, M.T)
    for _ in range(5):
        for M, R in zip(eng.one_body(), ref):
            assert np.array_equal(M, R)
