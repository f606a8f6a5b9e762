"""The tiled mixed build over occupied counts: each number of 16-wide column
chunks of the paired GEMM1, its remainders, the change to the single one (129
and more), fitted-function blocks of even and odd length, and counts that grow
and shrink within one engine's scratch, against the FP64 build.

Tolerance: the split-BF16 operands carry 16 bits or more and the products are
summed without cancellation of the largest elements: 1e-4 of the largest, the
bar of the other mixed tests; a column lost or counted twice moves K by about
1 / nocc.
"""
import numpy as np
import pytest

from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("waux", [0, 127, 1])
def test_tiled_mixed_columns(waux):
    from molecular2_b200.engine import IntegralEngine
    mol = geometry.water_cluster(4, 6.0, seed=4)
    obs = BasisSet(mol, "aug-cc-pvdz")
    eng = IntegralEngine(obs, BasisSet(mol, "avdz-jkfit"))
    eng.set_df_storage("tiled")
    eng.df_setup()
    eng.set_tiled_blocks(waux_max=waux)
    Q, _ = np.linalg.qr(np.random.default_rng(17).normal(size=(obs.nbf, obs.nbf)))
    counts = [20, 128] if waux == 1 else [144, 1, 16, 17, 33, 50, 64, 81, 97, 112, 113, 128, 129, 164]
    for nocc in counts:
        C = np.ascontiguousarray(Q[:, :nocc])
        J, K = eng.jk_df(C, 0)
        Jm, Km = eng.jk_df(C, 1)
        assert np.abs(Jm - J).max() < 1e-4 * np.abs(J).max(), nocc
        assert np.abs(Km - K).max() < 1e-4 * np.abs(K).max(), nocc
    eng.close()
