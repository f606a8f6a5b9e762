"""Engines on several threads at once whose launches of one kernel differ in
shared memory: RHF beside UHF builds, gradients of molecules of different
sizes, SCF runs of different matrix orders.  No call may fail and each gives
what it gives alone.

Tolerances: builds and gradients differ in the order of FP64 additions only
(elements <= 60, at most 1e5 terms a sum: 1e-11); SCF runs stop at a density
change of 1e-9, energies of size 400 then agree to 1e-9.
"""
import threading

import numpy as np
import pytest

from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet
from molecular2_b200.engine import IntegralEngine

pytestmark = pytest.mark.gpu


def waters(k, aux=None):
    mol = geometry.water_cluster(k, 3.5 * k ** (1 / 3), 5)
    return mol, BasisSet(mol, "cc-pvdz"), BasisSet(mol, aux) if aux else None


def orbitals(obs, k):
    return np.linalg.qr(np.random.default_rng(7).normal(size=(obs.nbf, 5 * k)))[0]


def rhf():
    _, obs, _ = waters(2)
    C, eng = orbitals(obs, 2), IntegralEngine(obs)
    return lambda: eng.jk_direct(2.0 * C @ C.T)


def uhf():
    _, obs, _ = waters(2)
    C, eng = orbitals(obs, 2), IntegralEngine(obs)
    return lambda: eng.jk_direct_uhf(C @ C.T, C[:, :7] @ C[:, :7].T)


def gradient(k):
    _, obs, aux = waters(k, "vdz-jkfit")
    C, eng = orbitals(obs, k), IntegralEngine(obs, aux)
    e = np.linspace(-1.0, -0.5, 5 * k)
    return lambda: [*eng.compute_forces(2.0 * C @ C.T, (C * e) @ C.T), *eng.compute_forces_df(C, e)]


def scf(k):
    mol, obs, aux = waters(k, "vdz-jkfit")
    eng = IntegralEngine(obs, aux)
    return lambda: [np.array(eng.scf_rhf(mol.nocc, mol.enuc(), df=True, densconverge=1e-9, enconverge=1e-9,
                                         guess="soad")[0].energy)]


def run(calls, repeats, tol):
    refs = [c() for c in calls]
    errors = []

    def work(call, ref):
        try:
            for _ in range(repeats):
                for got, want in zip(call(), ref):
                    assert np.abs(got - want).max() < tol * max(1.0, np.abs(want).max())
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=a) for a in zip(calls, refs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


@pytest.mark.parametrize("jobs,repeats,tol", [
    ([(rhf,), (uhf,), (rhf,), (uhf,)], 150, 1e-11),
    ([(gradient, 1), (gradient, 3), (gradient, 2)], 60, 1e-11),
    ([(scf, 4), (scf, 5), (scf, 6)], 12, 1e-9),
])
def test_calls_of_different_sizes_share_the_kernels(jobs, repeats, tol):
    run([f(*a) for f, *a in jobs], repeats, tol)


def one_shell(l, pair):
    """A single launch a build: one shell, RHF or UHF."""
    mol = geometry.water()
    obs = BasisSet.from_shells([(l, [0.8], [1.0], 0)], mol)
    eng, D = IntegralEngine(obs), np.eye(obs.nbf)
    return (lambda: eng.jk_direct_uhf(D, 0.5 * D)) if pair else (lambda: eng.jk_direct(D))


@pytest.mark.parametrize("l", [0, 1, 2])
def test_rhf_and_uhf_builds_of_one_class(l):
    run([one_shell(l, pair) for pair in (False, True, False, True)], 1500, 1e-13)
