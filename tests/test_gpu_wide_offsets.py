"""Level 0 in an order whose neighbours lie further apart than an int16 offset
reaches, on a level below and one above the size from which the outer
iteration's kernels change: nodes renumbered at random and loaded with their
operators.  The chained and the unchained solve give the same bits in either
precision, and the solution of the nodes' own order (to the solver's 1e-9)."""
import ctypes as C

import numpy as np
import pytest

import multigrid_meshless_b200 as mgm
from multigrid_meshless_b200 import _lib, api, clouds

pytestmark = pytest.mark.gpu


class Loaded(api.Multigrid):
    """A hierarchy loaded with its operators (mgm_load_level, mgm_prepare)."""

    def __init__(self, levels, dim, poly):
        self.L = _lib.load()
        self.nl, self.dim = len(levels), dim
        self.h = self.L.mgm_create(dim, 3, self.nl)
        self.sizes = []
        f, i = api._f, api._i
        for l, v in enumerate(levels):
            n, k = v["cloud"].shape
            a = [f(v[q]) for q in ("x", "y", "z", "nx", "ny", "nz")]
            _lib.check(self.L.mgm_load_level(self.h, l, n, int((v["btag"] != 0).sum()), *a, api._u8(v["btag"]), poly, k,
                                             i(v["cloud"]), f(v["Dx"]), f(v["Dy"]), None, f(v["lap"]), f(v["lapP"]),
                                             i(v["rpts"]), i(v["ppts"]), float(v["d_avg"])))
            self.sizes.append((n, 0, k, 0))
        _lib.check(self.L.mgm_prepare(self.h))


@pytest.mark.parametrize("m,k,poly", [(190, 20, 3), (190, 34, 4), (262, 20, 3)])
def test_neighbours_beyond_an_int16_offset(require_gpu, m, k, poly):
    rng = np.random.default_rng(m + k)
    mg = api.Multigrid(clouds.cavity_hierarchy(m, 3, seed=8), [k] * 3, [poly] * 3)
    levels = []
    for l in range(3):
        v = dict(mg.geometry(l))
        v.update({q: w for q, w in mg.operators(l).items() if w is not None})
        t = mg.transfer(l)
        v["rpts"], v["ppts"] = t["rpts"].copy(), t["ppts"].copy()
        levels.append(v)
    n = mg.n()
    b = np.cos(3 * levels[0]["x"]) * np.cos(2 * levels[0]["y"])
    b[levels[0]["btag"] != 0] = 0.0
    b[0] = 0.0
    mg.set_flow(Re=100.0, courant=0.3)
    mg.set_solver(rel_tol=1e-9, max_iters=100, cheb_degree=4, cheb_ratio=10.0)
    want = mg.solve_poisson(b, mode=mgm.MODE_FP64)[0]
    mg.close()
    # order[new] = old, node 0 (the pin) in its place
    order = np.concatenate([[0], 1 + rng.permutation(n - 1)])
    new = np.empty(n, np.int64)
    new[order] = np.arange(n)
    v = levels[0]
    for q in ("x", "y", "z", "nx", "ny", "nz", "btag", "Dx", "Dy", "lap", "lapP", "rpts", "ppts"):
        v[q] = np.ascontiguousarray(v[q][order])
    v["cloud"] = new[v["cloud"][order]].astype(np.int32)
    levels[1]["rpts"] = new[levels[1]["rpts"]].astype(np.int32)
    assert np.abs(v["cloud"] - np.arange(n)[:, None]).max() > 32767
    got = Loaded(levels, 2, poly)
    try:
        got.set_flow(Re=100.0, courant=0.3)
        got.set_solver(rel_tol=1e-9, max_iters=100, cheb_degree=4, cheb_ratio=10.0)
        for mode in (mgm.MODE_FP64, mgm.MODE_FP32_IR):
            out = []
            for graphs, chain in ((True, True), (False, True), (False, False)):
                got.use_graphs(graphs)
                got.use_launch_chaining(chain)
                out.append(got.solve_poisson(np.ascontiguousarray(b[order]), mode=mode))
            for p, it, rr in out:
                assert it == out[0][1] and np.array_equal(p, out[0][0]) and rr < 1e-9
            assert np.linalg.norm(out[0][0] - want[order]) <= 1e-6 * np.linalg.norm(want)
    finally:
        got.close()
