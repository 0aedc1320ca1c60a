"""A grid barrier's wait that runs out in a set-up kernel is reported as
MGM_ERR_TIMEOUT (built with no polls allowed, so that every CTA that has to wait
gives up at once), and the device works on."""
import ctypes as C

import numpy as np
import pytest

import probe
from multigrid_meshless_b200 import api

pytestmark = pytest.mark.gpu
MGM_ERR_TIMEOUT = 4


def test_set_up_kernels_report_a_timeout(require_gpu):
    L = probe.load("setup_probe", ["MGM_BARRIER_POLLS=0"])
    n, k = 600, 2
    p = lambda a: a.ctypes.data_as(C.c_void_p)
    idx = np.ascontiguousarray(np.stack([np.arange(n), (np.arange(n) + 1) % n]), dtype=np.int32)
    A = np.ascontiguousarray(np.stack([np.full(n, 4.0), np.ones(n)]))
    i64, i32 = np.zeros((n, n)), np.zeros((n, n), np.float32)
    assert L.probe_dense_inverse(n, k, p(idx), p(A), p(i64), p(i32), 148) == MGM_ERR_TIMEOUT
    n = 400000
    cloud = np.ascontiguousarray(np.stack([np.arange(n), (np.arange(n) + 1) % n, (np.arange(n) * 2) % n], axis=1),
                                 dtype=np.int32)
    q, reached = np.zeros(n, np.int32), C.c_int(0)
    assert L.probe_bfs_order(n, 3, p(cloud), p(q), C.byref(reached), 148) == MGM_ERR_TIMEOUT
    assert api.spmv(np.full((4, 2), 2.0), np.zeros((4, 2), np.int32), np.ones(4)).tolist() == [4.0] * 4
