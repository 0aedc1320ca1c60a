"""The set-up's cooperative kernels on other numbers of CTAs than one per SM of a
whole device: one, a few, and more than the device holds at once (the launch then
has what it does hold, where a grid of that size would be refused).  The bits do
not depend on the number."""
import ctypes as C

import numpy as np
import pytest

import probe

pytestmark = pytest.mark.gpu


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _inverse(n, k, idx, A, most):
    i64, i32 = np.zeros((n, n)), np.zeros((n, n), np.float32)
    rc = probe.load("setup_probe").probe_dense_inverse(n, k, _p(idx), _p(A), _p(i64), _p(i32), most)
    return rc, i64, i32


def _order(cloud, most):
    n, k = cloud.shape
    q, reached = np.zeros(n, np.int32), C.c_int(0)
    rc = probe.load("setup_probe").probe_bfs_order(n, k, _p(cloud), _p(q), C.byref(reached), most)
    return rc, reached.value, q


@pytest.mark.parametrize("n", [1, 7, 149, 700])
def test_inverse_on_any_number_of_ctas(require_gpu, n):
    k = min(n, 9)
    rng = np.random.default_rng(n)
    idx = np.stack([rng.permutation(n)[:k] for _ in range(n)], axis=1).astype(np.int32)  # [k][n]
    idx = np.ascontiguousarray(np.where(idx == np.arange(n), idx[0], idx))
    idx[0] = np.arange(n)
    A = rng.standard_normal((k, n))
    A[0] = 4.0 * k
    M = np.zeros((n, n))
    for j in range(k):
        np.add.at(M, (np.arange(n), idx[j]), A[j])
    rc, want, want32 = _inverse(n, k, idx, A, 148)
    assert rc == 0
    # a diagonally dominant system: forward error a few n times the rounding unit
    assert np.abs(want @ M - np.eye(n)).max() <= 16 * n * 2.0 ** -53
    assert np.array_equal(want32, want.astype(np.float32))
    for most in (1, 3, 64, 100000):
        rc, got, got32 = _inverse(n, k, idx, A, most)
        assert rc == 0 and np.array_equal(got, want) and np.array_equal(got32, want32), most


@pytest.mark.parametrize("n", [5, 10000, 2200000])
def test_order_on_any_number_of_ctas(require_gpu, n):
    # the largest: a grid by its size alone is more than the device holds
    i = np.arange(n, dtype=np.int64)
    cloud = np.stack([i, np.maximum(i - 1, 0), np.minimum(i + 1, n - 1), np.minimum(i * 2 + 1, n - 1)], axis=1)
    cloud = np.ascontiguousarray(cloud, dtype=np.int32)
    rc, reached, want = _order(cloud, 148)
    assert rc == 0 and reached == n and np.array_equal(np.sort(want), i)
    for most in (1, 5, 100000):
        rc, r, got = _order(cloud, most)
        assert rc == 0 and r == reached and np.array_equal(got, want), most
