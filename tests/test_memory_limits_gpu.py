"""Device memory: what a large fitted tensor takes, and calls that have to fit
into what is left.

The free memory is held by one torch tensor, down to a stated remainder.
"""
import numpy as np
import pytest

from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet
from molecular2_b200.engine import IntegralEngine, release_cached

pytestmark = pytest.mark.gpu
MB = 1 << 20


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


def system(k, basis="cc-pvdz", aux="vdz-jkfit"):
    mol = geometry.water_cluster(k, 3.5 * k ** (1 / 3), 5)
    obs, fit = BasisSet(mol, basis), BasisSet(mol, aux)
    C = np.linalg.qr(np.random.default_rng(7).normal(size=(obs.nbf, 5 * k)))[0]
    return mol, obs, fit, C


class leave:
    """All but `left` bytes of the device are held inside the block."""

    def __init__(self, left):
        self.left = left

    def __enter__(self):
        import torch
        release_cached()
        torch.cuda.empty_cache()
        self.t = torch.empty(free_bytes() - int(self.left), dtype=torch.uint8, device="cuda")

    def __exit__(self, *exc):
        import torch
        del self.t
        torch.cuda.empty_cache()


def tiled_engine(k):
    _, obs, fit, _ = system(k)
    eng = IntegralEngine(obs, fit)
    eng.set_df_storage("tiled")
    return eng


def test_large_blocks_take_what_they_hold():
    """Tiled split tensor of (H2O)18: two arrays of 652 MB.  Beside them the
    engine keeps the metric's two factors and, in at most 32 MB, its lists."""
    tiled_engine(2).df_setup()  # the kernels' code
    eng = tiled_engine(18)
    release_cached()
    before = free_bytes()
    eng.df_setup()
    release_cached()
    held = before - free_bytes()
    assert eng.df_tensor_bytes > 1 << 30
    assert held - eng.df_tensor_bytes - 2 * 8 * eng.naux ** 2 < 32 * MB


def test_df_gradient_in_the_memory_of_the_final_functions():
    """DF gradient on unpacked storage with room for X and W3 over the final
    functions (n = 160 against 180 Cartesian ones) and 16 MB: W3 over Cartesian
    functions does not fit and is made in blocks.  Sums in another order: 1e-10."""
    mol = geometry.water_cluster(4, 6.0, 5)
    shells = [(l, [x], [1.0], a) for a in range(0, 12, 3) for l, xs in ((2, (0.3, 0.6, 1.1, 2.5, 5.0)), (1, (0.4, 1.5)),
                                                                        (0, (0.2, 0.5, 1.2, 4.0, 12.0, 40.0, 150.0, 600.0, 3000.0)))
              for x in xs]
    obs = BasisSet.from_shells(shells, mol)
    fit = BasisSet(mol, "vdz-jkfit")
    n, o, naux = obs.nbf, 12, fit.nbf
    assert n == 160
    C = np.linalg.qr(np.random.default_rng(7).normal(size=(n, o)))[0]
    eps = np.linspace(-1.0, -0.5, o)
    eng = IntegralEngine(obs, fit)
    eng.set_df_storage("unpacked")
    eng.df_setup()
    ref = eng.compute_forces_df(C, eps)
    need = 8 * (n * naux * o + n * n * naux + 2 * o * o * naux + naux * naux)
    with leave(need + 16 * MB):
        got = eng.compute_forces_df(C, eps)
    for a, b in zip(got, ref):
        assert np.abs(a - b).max() < 1e-10 * max(1.0, np.abs(b).max())


def test_scf_when_the_free_memory_is_in_the_cache():
    """The first SCF of an engine makes the libraries' handles, which take device
    memory of their own: with 8 MB free and the rest in the library's cache it runs."""
    import torch
    mol, obs, _, _ = system(2)
    ref = IntegralEngine(obs).scf_rhf(mol.nocc, mol.enuc())[0].energy  # the libraries' code
    eng = IntegralEngine(obs)
    _, big, fit, C = system(8)
    other = IntegralEngine(big, fit)
    other.compute_forces_df(C, np.linspace(-1.0, -0.5, 40))
    other.close()
    torch.cuda.empty_cache()
    t = torch.empty(free_bytes() - 8 * MB, dtype=torch.uint8, device="cuda")
    r = eng.scf_rhf(mol.nocc, mol.enuc())[0]
    del t
    torch.cuda.empty_cache()
    assert r.converged and abs(r.energy - ref) < 1e-6
