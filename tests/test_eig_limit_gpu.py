"""SCF runs on both sides of the size up to which the Fock matrix is diagonalised
by the engine's own solver (160): six waters and three helium atoms, 159 functions,
with zero to two more s functions.

Tolerances as in test_small_eig_gpu.py: 1e-7 from a density change of 1e-9, 1e-11
for orthonormality.
"""
import numpy as np
import pytest

from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet, Molecule
from molecular2_b200.engine import IntegralEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("more", [0, 1, 2])
def test_scf_around_the_limit(more):
    from scipy.linalg import eigh
    w = geometry.water_cluster(6, 3.5 * 6 ** (1 / 3), 5)
    mol = Molecule(w.symbols + ["he"] * 3, np.vstack([w.xyz, [[20.0, 0.0, 0.0], [0.0, 20.0, 0.0], [0.0, 0.0, 22.0]]]),
                   angstrom=False)
    obs = BasisSet.from_shells(BasisSet(mol, "cc-pvdz").shells + [(0, [0.1], [1.0], 18 + k) for k in range(more)], mol)
    n = obs.nbf
    assert n == 159 + more
    eng = IntegralEngine(obs)
    r, x = eng.scf_rhf(mol.nocc, mol.enuc(), want=True, maxiter=60, densconverge=1e-9, enconverge=1e-9, guess="soad")
    assert r.converged
    S, T, V = eng.one_body()
    J, K = eng.jk_direct(x["D"], 1e-14)
    e, C = eigh(T + V + J - 0.5 * K, S)
    assert np.abs(e - x["eps"]).max() < 1e-7
    assert np.abs(2.0 * C[:, :mol.nocc] @ C[:, :mol.nocc].T - x["D"]).max() < 1e-7
    assert np.abs(x["C"].T @ S @ x["C"] - np.eye(n)).max() < 1e-11
