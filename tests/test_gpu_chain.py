"""The solver's chained kernels (operands fetched before the wait for the
predecessor) at the edges of their variants: stencils of every register chunk
(8, 24, 32, 40 slots and wider rows with a remainder), levels on either side
of the size from which the four-rows-per-thread and separate-reduction kernels
run, 2D and 3D.  Each solve must match an FP64 direct solve to the parity
bound of the other solver tests (1e-6), and graph replay, eager launches,
unchained launches and 32-bit indices must give the same bits (the sums of
every variant run in the same order)."""
import numpy as np
import pytest

import multigrid_meshless_b200 as mgm
from multigrid_meshless_b200 import api, clouds
from oracle import oracle as O

pytestmark = pytest.mark.gpu

CASES = [("cavity", 21, 2, 14, 2), ("cavity", 33, 2, 16, 3), ("cavity", 40, 2, 24, 3), ("cavity", 47, 2, 41, 4),
         ("cavity", 45, 2, 65, 4), ("cube", 13, 2, 35, 2), ("cavity", 255, 4, 30, 4), ("cavity", 257, 4, 30, 4)]


@pytest.mark.parametrize("shape,m,levels,k,poly", CASES)
def test_chained_kernels_at_their_edges(require_gpu, shape, m, levels, k, poly):
    make = clouds.cavity_hierarchy if shape == "cavity" else clouds.cube_hierarchy
    mg = api.Multigrid(make(m, levels, seed=31), [k] * levels, [poly] * levels)
    try:
        mg.set_solver(rel_tol=1e-9, max_iters=100, cheb_degree=4, cheb_ratio=10.0)
        g, ops = mg.geometry(0), mg.operators(0)
        b = np.cos(1.3 * np.pi * g["x"]) * np.cos(0.7 * np.pi * g["y"]) + 0.2 * np.sin(2 * g["z"])
        b[g["btag"] == 1] = 0.0
        b[0] = 0.0
        want = O.pinned_poisson_direct(ops["lapP"], g["cloud"], b)
        for mode in (mgm.MODE_FP64, mgm.MODE_FP32_IR):
            out = []
            for graphs, chain, compact in ((True, True, True), (False, True, True), (True, False, True),
                                           (True, True, False)):
                mg.use_graphs(graphs)
                mg.use_launch_chaining(chain)
                mg.use_compact(compact)
                out.append(mg.solve_poisson(b, mode=mode))
            mg.use_graphs(True), mg.use_launch_chaining(True), mg.use_compact(True)
            p, it, rr = out[0]
            assert rr < 1e-9
            assert np.linalg.norm(p - want) / np.linalg.norm(want) < 1e-6
            for p2, it2, _ in out[1:]:
                assert it2 == it and np.array_equal(p2, p)
    finally:
        mg.close()
