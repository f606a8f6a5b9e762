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
