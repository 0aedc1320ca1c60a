"""Contexts set up and solved in several threads at once (each with its own
stream; buffers from one pool, cooperative set-up kernels side by side) give the
bits of the same work one after the other."""
import threading

import numpy as np
import pytest

from multigrid_meshless_b200 import MODE_FP32_IR, api, clouds

pytestmark = pytest.mark.gpu


def _work(seed, out):
    fn, m, k, poly = ((clouds.cavity_hierarchy, 96, 20, 3), (clouds.cube_hierarchy, 24, 30, 2),
                      (clouds.cavity_hierarchy, 130, 30, 4))[seed % 3]
    for rep in range(2):
        mg = api.Multigrid(fn(m, 3, seed=seed), [k] * 3, [poly] * 3)
        try:
            mg.set_flow(Re=100.0, courant=0.3)
            mg.set_solver(rel_tol=1e-8, max_iters=80)
            g = mg.geometry(0)
            b = np.sin(3 * g["x"]) * np.cos(2 * g["y"])
            b[g["btag"] != 0] = 0.0
            b[0] = 0.0
            p, its, _ = mg.solve_poisson(b, mode=MODE_FP32_IR)
            out[seed, rep] = (g["cloud"], mg.operators(0)["lapP"], p, its)
        finally:
            mg.close()


def test_threads_give_the_bits_of_one(require_gpu):
    alone, together = {}, {}
    for s in range(6):
        _work(s, alone)
    ts = [threading.Thread(target=_work, args=(s, together)) for s in range(6)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert set(together) == set(alone)
    for key, want in alone.items():
        for a, b in zip(together[key], want):
            assert np.array_equal(a, b), key
