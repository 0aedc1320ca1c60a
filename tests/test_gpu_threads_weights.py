"""Operator rows of two stencils that one kernel instance serves, each asked for
over and over in threads of its own: the smaller stencil's launches must not
narrow what the larger one's may use.  One pair for the register kernels (orders
45 and 48) and one for the shared-memory kernels (71 and 81)."""
import threading

import numpy as np
import pytest

from multigrid_meshless_b200 import api, clouds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [((30, 4), (33, 4)), ((50, 5), (60, 5))])
def test_two_stencils_of_one_kernel(require_gpu, sizes):
    c = clouds.cavity2d(16, seed=4)
    jobs = []
    for k, poly in sizes:
        cloud = api.knn_cloud(c.x, c.y, c.z, c.btag, c.nb, k, 2)
        args = (c.x, c.y, c.z, c.nx, c.ny, c.nz, c.btag, cloud, 2, 3, poly)
        jobs.append((args, api.derivative_weights(*args)))
    bad = []

    def work(args, want):
        try:
            for _ in range(300):
                got = api.derivative_weights(*args)
                assert all(np.array_equal(got[q], want[q]) for q in ("Dx", "Dy", "lap", "lapP"))
        except Exception as e:
            bad.append(e)

    ts = [threading.Thread(target=work, args=j) for j in jobs * 2]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad[0]
