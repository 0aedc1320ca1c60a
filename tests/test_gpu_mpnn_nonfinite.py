"""Gradients that are infinite, not a number or next to the largest float: the
backward kernels give what the same products in FP32 give, an infinity where
those are infinite and a NaN only where those are."""
import numpy as np
import pytest

from test_gpu_mpnn_parts import CAT, H, ONE, _bf16, back, dW

pytestmark = pytest.mark.gpu
FLT_MAX = np.float32(3.4028235e38)


def _same(got, want, rel):
    assert np.array_equal(np.isnan(got), np.isnan(want))
    inf = np.isinf(want)
    assert np.array_equal(np.isinf(got), inf) and np.array_equal(got[inf], want[inf])
    fin = np.isfinite(want)
    assert np.all(np.abs(got[fin] - want[fin]) <= rel * np.abs(want[fin]))


def test_weight_gradient(require_gpu):
    n = 130
    rng = np.random.default_rng(4)
    dH = np.zeros((n, H), np.float32)
    dH[3, 0], dH[70, 1], dH[129, 2] = np.inf, -np.inf, np.nan
    dH[64, 3], dH[5, 4], dH[6, 5] = FLT_MAX, -FLT_MAX, np.float32(3.396e38)  # the last two round up beyond BF16's range
    dH[7, 6:] = rng.standard_normal(H - 6)
    cat = (rng.standard_normal((n, CAT)) * 2.0 ** -12).astype(np.float32)
    cat[:, ::5] = 0.0
    bits, c = _bf16(cat)
    with np.errstate(invalid="ignore"):
        want = np.array([[(c[:, q].astype(np.float64) * dH[:, f].astype(np.float64)).sum() for f in range(H)]
                         for q in range(CAT)])
    dz, _, gW = dW(dH, np.ones((n, H), np.float32), bits)
    assert np.array_equal(dz, dH, equal_nan=True)
    _same(gW, want, ONE)


def test_node_gradient(require_gpu):
    n, k = 70, 3
    rng = np.random.default_rng(5)
    dz = np.zeros((n, H), np.float32)
    dz[0, 3], dz[65, 9], dz[20, 11], dz[30, 12] = np.inf, -np.inf, np.nan, FLT_MAX
    W = (rng.standard_normal((H, CAT)) * 2.0 ** -12).astype(np.float32)
    W[:, ::7] = 0.0
    bits, w = _bf16(W)
    lap = np.full(n * k, 0.5, np.float32)
    src = [np.array([((j + 1) % n) * k]) for j in range(n)]
    d = dz.astype(np.float64)
    nb = d[(np.arange(n) + 1) % n]
    w = w.astype(np.float64)
    with np.errstate(invalid="ignore"):
        mul = lambda a, b: np.array([[(a[j] * b[:, q]).sum() for q in range(H)] for j in range(n)])
        want = mul(d, w[:, :H]) + mul(nb * float(np.float32(1) / np.float32(3)), w[:, H:2 * H]) + \
            mul(nb * 0.5, w[:, 2 * H:])
    got = back(k, src, lap, dz, bits, np.zeros((n, H), np.float32))
    _same(got, want, 2.0 ** -19)
