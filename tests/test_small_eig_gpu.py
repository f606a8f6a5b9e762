"""The SCF's own eigensolver for small matrices, over even and odd sizes up to
nearly its limit of 160 (2, 7, 25, 96, 120, 144, 150 functions):
orbital energies and the density of a converged run against numpy's
eigenproblem of the Fock matrix built from that density.

Tolerance: the run stops at a density change of 1e-9, which the Fock matrix
sees linearly (its elements are <= 40): 1e-7 for energies and densities; the
orbitals are orthonormal in S to n eps times the size of S^-1/2 (< 1e2): 1e-11.
"""
import numpy as np
import pytest

from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet, Molecule
from molecular2_b200.engine import IntegralEngine

pytestmark = pytest.mark.gpu

SYSTEMS = [
    ("h2", "sto-3g", True, 2), ("water1", "sto-3g", True, 7), ("water1", "cc-pvdz", False, 25),
    ("water4", "cc-pvdz", True, 96), ("water5", "cc-pvdz", True, 120),
    ("water6", "cc-pvdz", True, 144), ("water6", "cc-pvdz", False, 150),
]


@pytest.mark.parametrize("name,basis,spherical,n", SYSTEMS)
def test_scf_eigenpairs(name, basis, spherical, n):
    from scipy.linalg import eigh
    if name == "h2":
        mol = Molecule(["h", "h"], [[0.0, 0.0, 0.0], [0.0, 0.0, 0.74]])
    else:
        k = int(name[5:])
        mol = geometry.water_cluster(k, 3.5 * k ** (1 / 3), 5)
    obs = BasisSet(mol, basis, spherical=spherical)
    assert obs.nbf == n
    eng = IntegralEngine(obs)
    r, x = eng.scf_rhf(mol.nocc, mol.enuc(), want=True, maxiter=60, densconverge=1e-9, enconverge=1e-9, guess="soad")
    assert r.converged
    S, T, V = eng.one_body()
    J, K = eng.jk_direct(x["D"], 1e-14)
    e, C = eigh(T + V + J - 0.5 * K, S)
    assert np.abs(e - x["eps"]).max() < 1e-7
    assert np.abs(2.0 * C[:, :mol.nocc] @ C[:, :mol.nocc].T - x["D"]).max() < 1e-7
    assert np.abs(x["C"].T @ S @ x["C"] - np.eye(n)).max() < 1e-11
