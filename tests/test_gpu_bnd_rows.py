"""Boundary rows of the large levels (8 lanes a row) at stencil sizes around its
32- and 64-slot halves: the solve reaches its tolerance by the host's own FP64
residual, and a V-cycle whose boundary rows were solved wrongly would not: the
FP32 and FP64 preconditioners need the same number of V-cycles to within one,
with the boundary part inside the level's launch (2D) and before it (3D)."""
import numpy as np
import pytest
import scipy.sparse as sp

from multigrid_meshless_b200 import MODE_FP32_IR, MODE_FP64, api, clouds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,m,k,poly", [("cavity", 258, 31, 4), ("cavity", 258, 66, 5), ("cube", 41, 33, 2)])
def test_large_level_boundary_rows(require_gpu, shape, m, k, poly):
    fn = clouds.cavity_hierarchy if shape == "cavity" else clouds.cube_hierarchy
    mg = api.Multigrid(fn(m, 3, seed=2), [k] * 3, [poly] * 3)
    try:
        n = mg.n()
        assert n >= 65536
        mg.set_flow(Re=100.0, courant=0.3)
        mg.set_solver(rel_tol=1e-8, max_iters=80)
        g, ops = mg.geometry(0), mg.operators(0)
        rows = np.repeat(np.arange(n), k)
        A = sp.csr_matrix((ops["lapP"].ravel(), (rows, g["cloud"].ravel())), (n, n)).tolil()
        A[0, :] = 0.0
        A[0, 0] = 1.0
        A = A.tocsr()
        b = np.cos(2 * np.pi * g["x"]) * np.cos(np.pi * g["y"])
        b[g["btag"] != 0] = 0.0
        b[0] = 0.0
        its = {}
        for mode in (MODE_FP32_IR, MODE_FP64):
            p, its[mode], _ = mg.solve_poisson(b, mode=mode)
            assert np.linalg.norm(b - A @ p) <= 1.01e-8 * np.linalg.norm(b)
        assert abs(its[MODE_FP32_IR] - its[MODE_FP64]) <= 1
    finally:
        mg.close()
