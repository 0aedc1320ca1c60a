"""The network's backward kernels at node counts that do not fill their
64-node tiles, against the CPU oracle (same BF16 rounding points).  Oracle and
kernels round activations to BF16 from sums in different orders, so they part at
rounding ties: 20-node stencils agree to 2e-2 elsewhere in these tests, twice
that is allowed here.  The gradient of c_d, which passes no rounding, is checked
as the sum it is."""
import ctypes as C

import numpy as np
import pytest

from multigrid_meshless_b200 import _lib, api, clouds
from oracle import mpnn_oracle as MO

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [23, 41, 80])
def test_gradients_at_ragged_sizes(m):
    k, poly = 20, 3
    cl = clouds.cavity_hierarchy(m, 2, seed=9)
    mg = api.Multigrid(cl, [k, k], [poly, poly])
    try:
        L = _lib.load()
        _lib.check(L.mgm_mpnn_init(mg.h, 3, 0))
        _lib.check(L.mgm_mpnn_set_loss(mg.h, 1.0, 0.0))
        n, npar = mg.n(), L.mgm_mpnn_num_params()
        g = mg.geometry(0)
        f = [np.sin(a * g["x"] + b * g["y"]).astype(np.float32) for a, b in ((3, 1), (1, 4), (2, 2), (5, 3))]
        P = np.zeros(npar, np.float32)
        _lib.check(L.mgm_mpnn_params(mg.h, P.ctypes.data, None))
        grads, pred, loss = np.zeros(npar, np.float32), np.zeros(n, np.float32), C.c_double()
        _lib.check(L.mgm_mpnn_loss_grad(mg.h, *(a.ctypes.data for a in f), C.byref(loss), grads.ctypes.data,
                                        pred.ctypes.data))
        ops = mg.operators(0)
        G = MO.Graph(g["cloud"], (ops["lap"] * g["d_avg"] ** 2).astype(np.float32))
        feat = np.stack(f[:3] + [g["x"].astype(np.float32), g["y"].astype(np.float32),
                                 g["btag"].astype(np.float32)], axis=1)
        lo, go, _ = MO.loss_grad(P, feat, f[3], G, use_bf16=True)
        # sum of n FP32 terms of dy = 2 (y - t) / n: n * 2^-24 of the terms' absolute sum
        dy = 2.0 * (pred.astype(np.float64) - f[3]) / n
        assert abs(grads[MO.P_CD] - dy.sum()) <= n * 2.0 ** -24 * np.abs(dy).sum()
        assert abs(loss.value - np.mean((pred.astype(np.float64) - f[3]) ** 2)) <= 1e-6 * loss.value
        blocks = [(MO.P_WE, MO.P_CE), (MO.P_CE, MO.P_L0)]
        for l in range(MO.LAYERS):
            b = MO.P_L0 + l * MO.LAYER_PARAMS
            blocks += [(b, b + MO.CAT * MO.H), (b + MO.CAT * MO.H, b + MO.LAYER_PARAMS)]
        blocks += [(MO.P_WD, MO.P_CD)]
        for a, b in blocks:
            assert np.linalg.norm(grads[a:b] - go[a:b]) <= 4e-2 * np.linalg.norm(go[a:b]), (a, b)
    finally:
        mg.close()
