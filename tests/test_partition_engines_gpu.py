"""The partition of the direct builds across engines: every rank of a job has an
engine of its own, so the class lists must come out in the same order on each,
also where many pairs have the same Schwarz bound by symmetry.

Sums of partial builds differ from the whole in the order of the additions
only: elements <= 50 from <= 60^2 products, 1e-11 as in test_direct_jk_gpu.py.
"""
import numpy as np
import pytest

from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet, Molecule
from molecular2_b200.engine import IntegralEngine, JKError

pytestmark = pytest.mark.gpu


def chain(n, step=1.4):
    return Molecule(["h"] * n, [[0.0, 0.0, step * k] for k in range(n)], angstrom=False)


@pytest.mark.parametrize("obs", [
    BasisSet(geometry.water_cluster(2, 4.0, 3), "cc-pvdz"),
    BasisSet(geometry.water(), "cc-pvdz", spherical=False),
    BasisSet(geometry.alkane(3, 1), "6-311g**"),
    BasisSet(chain(12), "cc-pvdz"),
])
def test_schwarz_bounds_are_the_same_on_every_engine(obs):
    Q = IntegralEngine(obs).getPrescreen()
    for _ in range(5):
        assert np.array_equal(IntegralEngine(obs).getPrescreen(), Q)


def test_partial_builds_of_separate_engines_sum_to_the_whole():
    obs = BasisSet(chain(12), "cc-pvdz")
    rng = np.random.default_rng(5)
    D = rng.normal(size=(obs.nbf, obs.nbf))
    D = D + D.T
    eng = IntegralEngine(obs)
    J, K = eng.jk_direct(D, 1e-12)
    quartets = eng.last_quartets()
    g, _ = eng.compute_forces(D, 0.3 * D)
    scale = max(np.abs(J).max(), np.abs(K).max())
    for nranks in (2, 3):
        sJ, sK, sg, sq = np.zeros_like(J), np.zeros_like(K), np.zeros_like(g), 0
        for r in range(nranks):
            part = IntegralEngine(obs)
            part.set_direct_partition(r, nranks)
            j, k = part.jk_direct(D, 1e-12)
            sJ, sK, sq = sJ + j, sK + k, sq + part.last_quartets()
            sg += part.compute_forces(D, 0.3 * D)[0]
        assert sq == quartets
        assert max(np.abs(sJ - J).max(), np.abs(sK - K).max()) < 1e-11 * scale
        assert np.abs(sg - g).max() < 1e-10 * max(1.0, np.abs(g).max())


def many_kets():
    """Diffuse s shells, 2.2 million pairs, around one tight d shell: with the
    density on the d shell alone and this threshold only the (dd|ss) integrals
    pass the screen (bounds: dd about 5, ss 0.07, products 0.3 and 0.004)."""
    mol = Molecule(["he"], [[0.0, 0.0, 0.0]])
    shells = [(0, [float(x)], [1.0], 0) for x in np.linspace(1e-5, 2e-5, 2100)] + [(2, [1e3], [1.0], 0)]
    obs = BasisSet.from_shells(shells, mol)
    D = np.zeros((obs.nbf, obs.nbf))
    D[2100:, 2100:] = np.eye(5)
    return obs, D, 0.05


def test_no_class_is_left_out_of_a_build_without_an_error():
    """One bra pair and eight ranks: a launch that cannot be made is reported."""
    obs, D, precision = many_kets()
    eng = IntegralEngine(obs)
    J, _ = eng.jk_direct(D, precision)
    assert np.abs(J[:2100, :2100]).min() > 1e-3
    eng.set_direct_partition(0, 8)
    try:
        part, _ = eng.jk_direct(D, precision)
    except JKError:
        return
    assert np.abs(part - J)[:2100, :2100].max() < 1e-14


def test_fewer_bra_entries_than_ranks_with_many_kets():
    """The ket range of the (dd|ss) launch stays within the grid's limits."""
    obs, D, precision = many_kets()
    eng = IntegralEngine(obs)
    J, K = eng.jk_direct(D, precision)
    eng.set_direct_partition(0, 8)
    pJ, _ = eng.jk_direct(D, precision)
    assert np.abs(pJ - J)[:2100, :2100].max() < 1e-14
    uhf = eng.jk_direct_uhf(D, D, precision)
    assert np.abs(uhf[0] - J)[:2100, :2100].max() < 1e-14
