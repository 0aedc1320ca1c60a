"""Steps on levels of 65,536 rows and more (the level step waits on a device
counter inside its launch), a reference-mode cycle, a batched solve and training
samples side by side in threads, each several times: the bits of the same work
alone.  Training's gradients are FP32 atomic sums in no fixed order; they must
agree to 1e-5 of their norm, its loss and prediction bit for bit."""
import ctypes as C
import threading

import numpy as np
import pytest

from multigrid_meshless_b200 import BC_LID, MODE_FP32_IR, MODE_FP64, MODE_REFERENCE, _lib, api, clouds

pytestmark = pytest.mark.gpu


def _steps(fn, m, k, poly, mode, courant):
    mg = api.Multigrid(fn(m, 3, seed=6), [k] * 3, [poly] * 3, reference_transfer=mode == MODE_REFERENCE)
    try:
        assert mode == MODE_REFERENCE or mg.n() >= 65536
        mg.set_flow(Re=100.0, courant=courant, omega=0.25, num_relax=3, num_vcycles=5)
        mg.set_solver(rel_tol=1e-8, max_iters=80, cheb_degree=4, cheb_ratio=10.0)
        out = []
        for _ in range(3):
            mg.apply_bc(BC_LID)
            mg.run_steps(mode, 2)
            out += [mg.get_field("u"), mg.get_field("p")]
        return out
    finally:
        mg.close()


def _batch(mode):
    cl = clouds.shell_hierarchy(clouds.shell_h_for_nodes(12000), 2, seed=3)
    b = api.Batch(cl, [clouds.shell_stencil_sizes(cl[0], 40, 60), clouds.shell_stencil_sizes(cl[1], 25, 35)], [3, 2],
                  autotune=False)
    try:
        b.set_solver(rel_tol=1e-8, restart=24, cheb_degree=4, cheb_ratio=10.0)
        inner = b.level(0)["btag"] == 0
        f = np.random.default_rng(5).standard_normal((33, b.n()))
        f[:, ~inner] = 0.0
        f[:, inner] -= f[:, inner].mean(1, keepdims=True)
        f[:, 0] = 0.0
        return [np.array(b.solve(f, mode)[0]) for _ in range(3)]
    finally:
        b.close()


def _train():
    mg = api.Multigrid(clouds.cavity_hierarchy(120, 2, seed=9), [30] * 2, [4] * 2)
    try:
        L = _lib.load()
        _lib.check(L.mgm_mpnn_init(mg.h, 3, 0))
        g, n, npar = mg.geometry(0), mg.n(), L.mgm_mpnn_num_params()
        f = [np.sin(a * g["x"] + b * g["y"]).astype(np.float32) for a, b in ((3, 1), (1, 4), (2, 2), (5, 3))]
        out = []
        for _ in range(10):
            grads, pred, loss = np.zeros(npar, np.float32), np.zeros(n, np.float32), C.c_double()
            _lib.check(L.mgm_mpnn_loss_grad(mg.h, *(a.ctypes.data for a in f), C.byref(loss), grads.ctypes.data,
                                            pred.ctypes.data))
            out += [pred, grads]
        return out
    finally:
        mg.close()


WORK = {
    "cavity-fp32": lambda: _steps(clouds.cavity_hierarchy, 262, 30, 4, MODE_FP32_IR, 0.3),
    "cavity-fp64": lambda: _steps(clouds.cavity_hierarchy, 262, 30, 4, MODE_FP64, 0.3),
    "cube-fp32": lambda: _steps(clouds.cube_hierarchy, 41, 35, 2, MODE_FP32_IR, 0.1),
    "reference": lambda: _steps(clouds.cavity_hierarchy, 100, 20, 3, MODE_REFERENCE, 0.3),
    "batch-fp32": lambda: _batch(MODE_FP32_IR),
    "batch-fp64": lambda: _batch(MODE_FP64),
    "train": _train,
}


def test_side_by_side_as_alone(require_gpu):
    alone = {name: work() for name, work in WORK.items()}
    together, errors = {}, []

    def run(name):
        try:
            together[name] = WORK[name]()
        except Exception as e:
            errors.append((name, e))

    ts = [threading.Thread(target=run, args=(name,)) for name in WORK]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    for name, want in alone.items():
        for q, (a, b) in enumerate(zip(together[name], want, strict=True)):
            if name == "train" and q % 2:
                assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
            else:
                assert np.array_equal(a, b), (name, q)
