"""Gradients around the numbers of atoms up to which blocks sum them in shared
memory (512 in the two-electron kernels, 2,048 in the one-electron one): two
waters beside points of no charge and no basis function, which feel nothing
and change nothing but the path.

Sums in another order, elements <= 100: 1e-11.
"""
import numpy as np
import pytest

from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet, Molecule
from molecular2_b200.engine import IntegralEngine

pytestmark = pytest.mark.gpu


def gradients(natom):
    w = geometry.water_cluster(2, 4.0, 3)
    k = natom - w.natom
    points = np.stack([30.0 + np.arange(k) % 50, 30.0 + np.arange(k) // 50 % 50, 30.0 + np.arange(k) // 2500], axis=1)
    mol = Molecule(w.symbols + ["h"] * k, np.vstack([w.xyz, points]), angstrom=False)
    mol.Z[w.natom:] = 0.0
    obs, aux = (BasisSet.from_shells(BasisSet(w, b).shells, mol) for b in ("cc-pvdz", "vdz-jkfit"))
    C = np.linalg.qr(np.random.default_rng(4).normal(size=(obs.nbf, 10)))[0]
    e = np.linspace(-1.0, -0.5, 10)
    eng = IntegralEngine(obs, aux)
    return [*eng.compute_forces(2.0 * C @ C.T, (C * e) @ C.T), *eng.compute_forces_df(C, e)]


@pytest.fixture(scope="module")
def alone():
    return gradients(6)


@pytest.mark.parametrize("natom", [512, 513, 2048, 2049])
def test_gradients_with_many_atoms(natom, alone):
    for got, ref in zip(gradients(natom), alone):
        assert np.abs(ref).max() < 100.0
        assert np.abs(got[:6] - ref).max() < 1e-11
        assert not got[6:].any()
