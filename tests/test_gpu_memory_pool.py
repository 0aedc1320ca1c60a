"""The library's device-memory pool keeps at most 2 GiB beyond the buffers in
use when a call returns: after a stand-alone call with 3 GiB of temporaries, after
a context shrinks its Krylov space, after a call that fails with its buffers
allocated, and after the context is gone."""
import numpy as np
import pytest

from multigrid_meshless_b200 import _lib, api, clouds

pytestmark = pytest.mark.gpu
KEPT = (2 << 30) + (64 << 20)  # the bound and the pool's granularity


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_idle_memory_is_bounded(require_gpu):
    api.spmv(np.ones((4, 2)), np.zeros((4, 2), np.int32), np.ones(4))
    before = _free()
    n, k = 2_000_000, 64
    D = np.zeros((n, k))
    cloud = np.zeros((n, k), np.int32)
    f = np.ones(n)
    assert np.all(api.spmv(D, cloud, f) == 0.0)
    assert before - _free() <= KEPT
    # a refused call keeps no more
    cloud[-1, -1] = n
    with pytest.raises(_lib.MgmError):
        api.spmv(D, cloud, f)
    assert before - _free() <= KEPT
    del D, cloud, f


def test_a_context_gives_back_what_it_no_longer_needs(require_gpu):
    start = _free()
    mg = api.Multigrid(clouds.cavity_hierarchy(1440, 6, seed=2), [12] * 6, [2] * 6)
    try:
        mg.set_solver(rel_tol=1e-8, max_iters=8)
        small = _free()
        mg.set_solver(rel_tol=1e-8, max_iters=128)   # 20 bytes a node and vector: 4.9 GiB
        mg.set_solver(rel_tol=1e-8, max_iters=127)   # freed and allocated again
        assert small - _free() <= 20 * 129 * mg.n() + KEPT
        mg.set_solver(rel_tol=1e-8, max_iters=8)
        assert small - _free() <= KEPT
    finally:
        mg.close()
    assert start - _free() <= KEPT
