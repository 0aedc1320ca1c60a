"""A context that one thread worked on last and another destroys: the first
thread's next calls, one with buffers large enough that the pool is trimmed, do not
use the stream that went with it."""
import threading

import numpy as np
import pytest

from multigrid_meshless_b200 import MODE_FP64, api, clouds

pytestmark = pytest.mark.gpu


def test_context_destroyed_in_another_thread(require_gpu):
    box, errors = {}, []
    used, gone = threading.Event(), threading.Event()

    def worker():
        try:
            mg = box["mg"] = api.Multigrid(clouds.cavity_hierarchy(40, 2, seed=3), [20] * 2, [3] * 2)
            mg.set_flow(Re=100.0, courant=0.3)
            b = np.zeros(mg.n())
            b[mg.geometry(0)["btag"] == 0] = 1.0
            b[0] = 0.0
            mg.set_solver(rel_tol=1e-8, max_iters=60)
            mg.solve_poisson(b, mode=MODE_FP64)
            used.set()
            gone.wait(60)
            n, k = 400000, 30
            one = np.ones((n, k))
            out = api.laplacian_for_poisson(one, one, None, 2 * one, np.ones(n), np.zeros(n), None, np.zeros(n, np.uint8))
            assert np.array_equal(out, 2 * one)
            box["cloud"] = api.knn_cloud(*(np.random.default_rng(1).random((2, 5000))), np.zeros(5000),
                                         np.zeros(5000, np.uint8), 0, 12, 2)
        except Exception as e:
            errors.append(e)
            used.set()

    t = threading.Thread(target=worker)
    t.start()
    assert used.wait(120)
    if "mg" in box:
        box.pop("mg").close()
    gone.set()
    t.join()
    assert not errors, errors[0]
    assert np.array_equal(box["cloud"][:, 0], np.arange(5000))
