"""FP64 DF builds over occupied counts around every tile width of the FP64 GEMM
(and odd function counts, whose rows are only 8-byte aligned), against the
oracle; both storages, so row- and column-contiguous operands.

Tolerance: K sums naux * nocc <= 117 * 130 products of size <= 2 in another
order, 2 * 15,210 * 1.1e-16 = 3e-12 at worst; 1e-11 leaves a factor three.
"""
import numpy as np
import pytest

import oracle
from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet
from molecular2_b200.engine import IntegralEngine

pytestmark = pytest.mark.gpu
NOCC = [1, 8, 15, 16, 17, 31, 32, 33, 40, 41, 48, 49, 64, 65, 80, 81, 96, 97, 128, 129, 130]


@pytest.mark.parametrize("odd", [False, True])
def test_df_build_over_tile_widths(odd):
    mol = geometry.water()
    obs, aux = BasisSet(mol, "cc-pvdz"), BasisSet(mol, "vdz-jkfit")
    if odd:
        obs = BasisSet.from_shells(obs.shells[:-1], mol)
        aux = BasisSet.from_shells([s for i, s in enumerate(aux.shells) if i != 9], mol)
        assert obs.nbf % 2 == 1 and aux.nbf % 2 == 1
    B = oracle.df_B(oracle.eri3(obs, aux), oracle.eri2(aux))
    engines = []
    for storage in ("unpacked", "tiled"):
        e = IntegralEngine(obs, aux)
        e.set_df_storage(storage)
        e.df_setup()
        engines.append(e)
    rng = np.random.default_rng(11)
    for nocc in NOCC:
        C = rng.normal(size=(obs.nbf, nocc)) / np.sqrt(nocc)
        Jr, Kr = oracle.df_jk(B, C)
        assert max(np.abs(Jr).max(), np.abs(Kr).max()) < 40.0
        for e in engines:
            J, K = e.jk_df(C)
            assert max(np.abs(J - Jr).max(), np.abs(K - Kr).max()) < 1e-11, (nocc, e.df_storage)
