"""FP64 build on tiled storage with Y = L^-1 X' in row batches copied back over X'
(a capped occupied slice) against Y kept whole, for one slice, several of unequal
width and 65 rows (one more than a batch).

J and K are sums of n naux o products in another order: 1e-11 of their size.
"""
import numpy as np
import pytest

from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet
from molecular2_b200.engine import IntegralEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,extra,nocc,cap", [(1, 0, 5, 5), (1, 0, 5, 2), (2, 17, 10, 10), (6, 0, 30, 7), (6, 0, 30, 30)])
def test_row_batches(k, extra, nocc, cap):
    mol = geometry.water_cluster(k, 3.5 * k ** (1 / 3), 5)
    shells = BasisSet(mol, "cc-pvdz").shells + [(0, [0.2 + 0.3 * j], [1.0], j % mol.natom) for j in range(extra)]
    obs, aux = BasisSet.from_shells(shells, mol), BasisSet(mol, "vdz-jkfit")
    C = np.linalg.qr(np.random.default_rng(1).normal(size=(obs.nbf, nocc)))[0]
    eng = IntegralEngine(obs, aux)
    eng.set_df_storage("tiled")
    eng.df_setup()
    ref = eng.jk_df(C)
    eng.set_tiled_blocks(oc_max=cap)
    for got, want in zip(eng.jk_df(C), ref):
        assert np.abs(got - want).max() < 1e-11 * np.abs(want).max()
