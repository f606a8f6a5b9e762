"""The cache of freed device blocks: memory comes back, stays bounded, and
engines on several threads that share it give the results of one alone.

The thread test compares builds of the same inputs: only the order of FP64
atomic additions differs, 24 x 24 sums of size <= 10: 1e-12.
"""
import threading
import time

import numpy as np
import pytest

from molecular2_b200 import geometry
from molecular2_b200.basis import BasisSet
from molecular2_b200.engine import IntegralEngine, release_cached

pytestmark = pytest.mark.gpu


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


def one_geometry(seed):
    mol = geometry.water_cluster(1, 3.5, seed)
    obs, aux = BasisSet(mol, "cc-pvdz"), BasisSet(mol, "vdz-jkfit")
    C = np.linalg.qr(np.random.default_rng(seed).normal(size=(obs.nbf, 5)))[0]
    eng = IntegralEngine(obs, aux)
    eng.df_setup()
    out = [*eng.jk_df(C), *eng.jk_direct(2.0 * C @ C.T), *eng.compute_forces_df(C, np.linspace(-1.0, -0.5, 5))]
    eng.close()
    return out


def test_cached_memory_is_bounded_and_given_back():
    one_geometry(1)
    release_cached()
    before = free_bytes()
    for seed in range(4):
        one_geometry(seed)
        assert before - free_bytes() <= 4 << 30
    release_cached()
    assert abs(before - free_bytes()) <= 64 << 20  # code modules loaded meanwhile


def test_threads_share_the_cache():
    refs = [one_geometry(s) for s in range(6)]
    got, errors = {}, []

    def work(ids):
        try:
            for s in ids:
                got[s] = one_geometry(s)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(ids,)) for ids in ([0, 1], [2, 3], [4, 5])]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for s, ref in enumerate(refs):
        for a, b in zip(got[s], ref):
            assert np.abs(a - b).max() < 1e-12


def test_allocations_do_not_wait_for_a_free_on_another_thread():
    """A free waits for the device; meanwhile another thread's call that needs
    memory and only queues work comes back."""
    import torch
    mol = geometry.water_cluster(1, 3.5, 1)
    obs = BasisSet(mol, "cc-pvdz")
    D = torch.eye(obs.nbf, dtype=torch.float64, device="cuda")
    J, K = torch.empty_like(D), torch.empty_like(D)
    warm = IntegralEngine(obs)
    warm.jk_direct_device(D.data_ptr(), J.data_ptr(), K.data_ptr())  # the kernels' code
    warm.close()
    going, fresh = IntegralEngine(obs), IntegralEngine(obs)
    side, done = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(2_000_000_000)  # about a second
        done.record()
    t = threading.Thread(target=going.close)
    t.start()
    time.sleep(0.2)  # close() is in its first free
    assert t.is_alive()
    fresh.jk_direct_device(D.data_ptr(), J.data_ptr(), K.data_ptr())
    assert not done.query()
    t.join()
    torch.cuda.synchronize()
