"""Batched solve at the edges of its kernels' ranges: either row shape (few rows
per CTA, or all rows split among two CTAs per SM), either width (32 or 64
columns), row lengths that are no multiple of the chunk, and coarsest levels
that are no multiple of the dense product's tile.  Every right-hand side solves
the pinned FP64 system (residual from the host below the requested 1e-8 plus
1e-10 for rounding) and the FP32 preconditioner costs at most one V-cycle more
than the FP64 one."""
import numpy as np
import pytest
import scipy.sparse as sp

from multigrid_meshless_b200 import MODE_FP32_IR, MODE_FP64, api, clouds

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes,levels,k,nrhs", [(1700, 2, 31, 1), (3100, 2, 45, 32), (13500, 3, 37, 33),
                                                  (16000, 3, 50, 64)])
def test_batched_rows(nodes, levels, k, nrhs):
    cl = clouds.shell_hierarchy(clouds.shell_h_for_nodes(nodes), levels, seed=3)
    ks = [clouds.shell_stencil_sizes(cl[0], k, k + 7)] + [clouds.shell_stencil_sizes(c, 25, 35) for c in cl[1:]]
    b = api.Batch(cl, ks, [3] + [2] * (levels - 1), phs=3, autotune=False)
    try:
        b.set_solver(rel_tol=1e-8, restart=24, cheb_degree=4, cheb_ratio=10.0)
        lev = b.level(0)
        n = len(lev["x"])
        A = sp.csr_matrix((lev["lapP"].copy(), lev["col"].astype(np.int64), lev["row_ptr"].astype(np.int64)), (n, n))
        A.data[A.indptr[0]:A.indptr[1]] = np.where(A.indices[A.indptr[0]:A.indptr[1]] == 0, 1.0, 0.0)
        inner = lev["btag"] == 0
        f = np.random.default_rng(5).standard_normal((nrhs, n))
        f[:, ~inner] = 0.0
        f[:, inner] -= f[:, inner].mean(1, keepdims=True)
        f[:, 0] = 0.0
        cycles = {}
        for mode in (MODE_FP32_IR, MODE_FP64):
            sol, cycles[mode], rr, _ = b.solve(f, mode)
            res = f.T - A @ np.asarray(sol).T
            assert np.all(np.linalg.norm(res, axis=0) <= (1e-8 + 1e-10) * np.linalg.norm(f, axis=1))
        assert cycles[MODE_FP32_IR] <= cycles[MODE_FP64] + 1
    finally:
        b.close()
