"""The set-up's cooperative kernels at the edges of their ranges: breadth-first
order on graphs of many tiny levels, of a few huge ones and of one node; the
coarsest inverse with its rows in shared memory and, above about 1800 rows, in
global memory."""
import numpy as np
import pytest

from multigrid_meshless_b200 import MODE_FP64, api, clouds

pytestmark = pytest.mark.gpu


def _fifo(cloud):
    """The queue of a breadth-first walk from node 0, slots 1.. in order."""
    n, seen, q = len(cloud), {0}, [0]
    for i in q:
        for c in cloud[i, 1:]:
            if c not in seen:
                seen.add(c)
                q.append(c)
    return np.array(q, np.int32) if len(q) == n else None


def _graph(kind, n, rng):
    own = np.arange(n)[:, None]
    if kind == "chain":      # one node a level
        return np.hstack([own, np.minimum(own + 1, n - 1)]).astype(np.int32)
    if kind == "tree":       # levels of 1, 40, 1600, ... nodes
        ch = np.minimum(40 * own + 1 + np.arange(40)[None, :], n - 1)
        return np.hstack([own, ch]).astype(np.int32)
    perm = rng.permutation(n)  # a shuffled ring plus random edges
    nxt = np.empty(n, np.int64)
    nxt[perm] = np.roll(perm, -1)
    return np.hstack([own, nxt[:, None], rng.integers(0, n, (n, 5))]).astype(np.int32)


@pytest.mark.parametrize("kind,n", [("chain", 1), ("chain", 700), ("tree", 100_000), ("tree", 4097), ("random", 300),
                                     ("random", 50_001), ("random", 400_000)])
def test_bfs_order(require_gpu, kind, n):
    cloud = _graph(kind, n, np.random.default_rng(n))
    assert np.array_equal(api.bfs_order(cloud), _fifo(cloud))


@pytest.mark.parametrize("m", [12, 13, 42, 45])
def test_one_level_solve_is_direct(require_gpu, m):
    """On a single level the V-cycle is the inverse of the pinned operator: the
    FP64 solve takes one V-cycle (two where the operator's condition, about m^2
    times 10, leaves more than 1e-11 of the right-hand side)."""
    mg = api.Multigrid(clouds.cavity_hierarchy(m, 1, seed=4), [20], [3])
    try:
        assert mg.n() <= 8192
        mg.set_flow(Re=100.0, courant=0.5)
        mg.set_solver(rel_tol=1e-11, max_iters=10)
        b = np.random.default_rng(m).standard_normal(mg.n())
        b[mg.geometry(0)["btag"] != 0] = 0.0
        b[0] = 0.0
        _, its, rr = mg.solve_poisson(b, mode=MODE_FP64)
        assert its <= 2 and rr < 1e-11
    finally:
        mg.close()
