"""The backward kernels' three-part split of the FP32 gradients, on given arrays
against 64-bit products, at node counts that leave a partial tile and with
several tiles per CTA.

Two checks of each product.  One term: an output that is one gradient times a
power of two must come back to 2^-21 relative (two truncations of 2^-23 and a
margin of two); the largest part alone is off by up to 2^-9, the two largest by
up to 2^-17.  All terms: |error| <= steps * 2^-23 * sum |a||b|, steps the
accumulation steps an output goes through (16 products a step, three parts, then
the tiles and the CTAs)."""
import ctypes as C

import numpy as np
import pytest

import probe

gpu = pytest.mark.gpu
H, CAT, TILE, CTAS = 64, 192, 64, 148
ONE = 2.0 ** -21


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _bf16(x):
    """Round to BF16 (ties to even): (bits, value)."""
    u = np.ascontiguousarray(x, np.float32).view(np.uint32)
    b = ((u + 0x7FFF + ((u >> 16) & 1)) >> 16).astype(np.uint16)
    return b, (b.astype(np.uint32) << 16).view(np.float32)


def _gradients(rng, shape):
    # full significands over four decades
    return (rng.standard_normal(shape) * 10.0 ** rng.uniform(-4, 0, shape)).astype(np.float32)


def dW(dH, z, cat):
    n = len(dH)
    dz, gb, gW = np.zeros((n, H), np.float32), np.zeros(H, np.float32), np.zeros((CAT, H), np.float32)
    assert probe.load("mpnn_probe").probe_dW(n, _p(dH), _p(z), _p(cat), _p(dz), _p(gb), _p(gW)) == 0
    return dz, gb, gW


def back(k, src, lap, dz, WT, dH):
    """src: per node j the positions i * k + slot of its in-edges, a list."""
    n = len(dz)
    ptr = np.zeros(n + 1, np.int32)
    ptr[1:] = np.cumsum([len(s) for s in src])
    pos = np.concatenate([np.asarray(s, np.int32) for s in src] + [np.zeros(1, np.int32)]).astype(np.int32)
    out = dH.copy()
    assert probe.load("mpnn_probe").probe_back(n, k, len(pos), _p(ptr), _p(pos), _p(lap), _p(dz), _p(WT), _p(out)) == 0
    return out


def test_the_bound_tells_the_parts_apart():
    # on the host: three parts give the value back, two miss the one-term bound nearly always
    v = _gradients(np.random.default_rng(1), 4096)
    sums, r = [], v.copy()
    for _ in range(3):
        part = _bf16(r)[1]
        r = r - part
        sums.append((sums[-1] if sums else 0.0) + part.astype(np.float64))
    assert np.array_equal(sums[2], v.astype(np.float64))
    for two in sums[:2]:
        assert np.mean(np.abs(two - v) > ONE * np.abs(v)) > 0.5


@gpu
@pytest.mark.parametrize("n", [1, 63, 65, 193, CTAS * TILE + 100])
def test_weight_gradient_against_64_bits(require_gpu, n):
    rng = np.random.default_rng(n)
    dH = _gradients(rng, (n, H))
    z = rng.standard_normal((n, H)).astype(np.float32)
    cat_bits, cat = _bf16(rng.standard_normal((n, CAT)))
    want = np.where(z > 0, dH, np.float32(0))
    dz, gb, gW = dW(dH, z, cat_bits)
    assert np.array_equal(dz, want)
    steps = 12 + 2 * -(-n // (TILE * CTAS)) + CTAS
    w64, c64 = want.astype(np.float64), cat.astype(np.float64)
    assert np.all(np.abs(gW - c64.T @ w64) <= steps * 2.0 ** -23 * (np.abs(c64).T @ np.abs(w64)))
    rows = -(-n // 32) + 32 + CTAS
    assert np.all(np.abs(gb - w64.sum(0)) <= rows * 2.0 ** -24 * np.abs(w64).sum(0))
    # one node per output row: a gradient times a power of two
    node = (np.arange(CAT) * 37) % n
    one = np.zeros((n, CAT), np.float32)
    one[node, np.arange(CAT)] = 2.0 ** rng.integers(-8, 8, CAT)
    _, _, gW = dW(dH, np.ones_like(z), _bf16(one)[0])
    exact = dH[node].astype(np.float64) * one[node, np.arange(CAT)].astype(np.float64)[:, None]
    assert np.all(np.abs(gW - exact) <= ONE * np.abs(exact))


@gpu
@pytest.mark.parametrize("n,k", [(1, 3), (63, 7), (130, 30), (1000, 30)])
def test_node_gradient_against_64_bits(require_gpu, n, k):
    rng = np.random.default_rng(n + k)
    dz = _gradients(rng, (n, H))
    lap = rng.standard_normal(n * k).astype(np.float32)
    order = rng.permutation(n * k)
    # in-degrees from 0 to beyond a gather's 16 edges
    cuts = np.sort(rng.integers(0, n * k + 1, n - 1))
    src = np.split(order, cuts)
    dH = _gradients(rng, (n, H))
    bits, WT = _bf16(rng.standard_normal((H, CAT)) / 8)
    got = back(k, src, lap, dz, bits, dH)
    d64, w64 = dz.astype(np.float64), WT.astype(np.float64)
    s1 = np.array([d64[s // k].sum(0) for s in src]) / k
    s2 = np.array([(lap[s].astype(np.float64)[:, None] * d64[s // k]).sum(0) for s in src])
    want = dH + d64 @ w64[:, :H] + s1 @ w64[:, H:2 * H] + s2 @ w64[:, 2 * H:]
    a1 = np.array([np.abs(d64[s // k]).sum(0) for s in src]) / k
    a2 = np.array([np.abs(lap[s].astype(np.float64)[:, None] * d64[s // k]).sum(0) for s in src])
    size = np.abs(dH) + np.abs(d64) @ np.abs(w64[:, :H]) + a1 @ np.abs(w64[:, H:2 * H]) + a2 @ np.abs(w64[:, 2 * H:])
    deg = max(len(s) for s in src)
    assert np.all(np.abs(got - want) <= (12 + 4 + deg) * 2.0 ** -23 * size)
    # one block of the weights at a time, one feature per output, one in-edge per node
    src1 = [np.array([((j * 13) % n) * k + j % k]) for j in range(n)]
    e = np.array([s[0] for s in src1])
    x = [dz, (dz[e // k] * np.float32(1.0 / k)).astype(np.float32), (lap[e][:, None] * dz[e // k]).astype(np.float32)]
    for part in range(3):
        W1 = np.zeros((H, CAT), np.float32)
        f = rng.permutation(H)
        W1[f, part * H + np.arange(H)] = 2.0 ** rng.integers(-8, 8, H)
        got = back(k, src1, lap, dz, _bf16(W1)[0], np.zeros_like(dH))
        exact = x[part][:, f].astype(np.float64) * W1[f, part * H + np.arange(H)].astype(np.float64)
        assert np.all(np.abs(got - exact) <= ONE * np.abs(exact))
