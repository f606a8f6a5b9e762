"""Three- and two-index integrals and the DF gradient for every kind of fitting
shell (s, p, pure and Cartesian d and f) and for contracted ones, against the
oracle.

Tolerances: an integral of size <= 40 sums at most 64 x 9 primitive terms,
40 * sqrt(576) * 1.1e-16 = 1e-13, 1e-12 leaves a factor ten for the terms'
cancellation.  The gradient goes through V^-1: its rounding is bounded by
cond(V) eps times its size, times the number of terms' root (~50).
"""
import numpy as np
import pytest

import oracle
from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet
from molecular2_b200.engine import IntegralEngine

pytestmark = pytest.mark.gpu


def shell(l, n, atom, lo, hi):
    exps = np.geomspace(hi, lo, n) if n > 1 else np.array([lo])
    return (l, [float(x) for x in exps], [float(0.4 + 0.2 * k) for k in range(n)], atom)


def systems(spherical_aux, mixed_lengths):
    mol = geometry.water()
    obs = BasisSet.from_shells([shell(0, 8, 0, 0.3, 60.0), shell(1, 2, 0, 0.4, 3.0), shell(2, 1, 0, 0.8, 1.0),
                                shell(0, 1, 1, 0.5, 1.0), shell(1, 1, 2, 0.7, 1.0), shell(2, 1, 2, 1.1, 1.0)], mol,
                               spherical=mixed_lengths)
    k = 3 if mixed_lengths else 1
    aux = BasisSet.from_shells([shell(0, k, 0, 0.4, 9.0), shell(1, 1, 0, 0.9, 1.0), shell(2, k, 0, 0.7, 4.0),
                                shell(3, 1, 0, 1.0, 1.0), shell(0, 1, 1, 0.6, 1.0), shell(1, k, 1, 0.5, 3.0),
                                shell(2, 1, 2, 0.8, 1.0), shell(3, k, 2, 0.9, 4.0)], mol, spherical=spherical_aux)
    return obs, aux


@pytest.mark.parametrize("spherical_aux", [True, False])
@pytest.mark.parametrize("mixed_lengths", [True, False])
def test_fitting_shell_kinds(spherical_aux, mixed_lengths):
    obs, aux = systems(spherical_aux, mixed_lengths)
    eng = IntegralEngine(obs, aux)
    T, V = eng.compute_eris_3index(), eng.compute_eris_2index()
    Tr, Vr = np.asarray(oracle.eri3(obs, aux)), oracle.eri2(aux)
    assert max(np.abs(Tr).max(), np.abs(Vr).max()) < 40.0
    assert np.abs(V - Vr).max() < 1e-12
    assert np.abs(T - Tr).max() < 1e-12
    C = np.random.default_rng(5).normal(size=(obs.nbf, 3)) * 0.3
    eps = np.array([-1.0, -0.6, -0.3])
    ref = oracle.df_grad2e(obs, aux, C)
    tol = 50 * 1.1e-16 * np.linalg.cond(Vr) * max(1.0, np.abs(ref).max())
    assert tol < 1e-9
    for storage in ("unpacked", "tiled"):
        e = IntegralEngine(obs, aux)
        e.set_df_storage(storage)
        e.df_setup()
        _, g2 = e.compute_forces_df(C, eps)
        assert np.abs(g2 - ref).max() < tol
        J, K = e.jk_df(C)
        Jr, Kr = oracle.df_jk(oracle.df_B(Tr, Vr), C)
        assert max(np.abs(J - Jr).max(), np.abs(K - Kr).max()) < tol
