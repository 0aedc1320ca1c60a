"""The weight solves with the system in registers: orders at the edges of every
register size (multiples of four and one beyond), 2D and 3D, up to the largest
(64) and one above it (the shared-memory kernel), other RBF exponents, a
polynomial degree above the table of powers.  Bit for bit against the
correctly-rounded-power oracle, as the other set-up tests."""
import numpy as np
import pytest

from multigrid_meshless_b200 import api, clouds
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# dim, k, poly, phs -> order k + np
CASES = [(2, 9, 1, 3), (2, 13, 1, 3), (2, 14, 1, 3), (2, 18, 3, 3), (2, 19, 3, 5), (2, 22, 3, 3), (2, 23, 3, 3),
         (2, 30, 4, 3), (2, 33, 4, 3), (2, 34, 4, 7), (2, 49, 4, 3), (2, 50, 4, 3), (2, 12, 0, 3),
         (3, 25, 2, 3), (3, 35, 2, 5), (3, 38, 2, 3), (3, 39, 2, 3), (3, 44, 3, 3)]


@pytest.mark.parametrize("dim,k,poly,phs", CASES)
def test_weights_bit_exact_at_register_sizes(require_gpu, dim, k, poly, phs):
    make = (lambda m, s: clouds.cavity2d(m, seed=s)) if dim == 2 else (lambda m, s: clouds.cube3d(m, seed=s))
    F, C = make(17 if dim == 2 else 8, 11), make(13 if dim == 2 else 7, 12)
    fs, cs = O.orc_level_setup(F, k), O.orc_level_setup(C, k)
    got = api.derivative_weights(fs["x"], fs["y"], fs["z"], fs["nx"], fs["ny"], fs["nz"], fs["btag"], fs["cloud"], dim,
                                 phs, poly)
    want = [np.zeros(F.n * k) for _ in range(5)]
    O.lib(True).orc_derivative_weights(F.n, k, dim, phs, poly, fs["x"], fs["y"], fs["z"], fs["nx"], fs["ny"], fs["nz"],
                                       fs["btag"], np.ascontiguousarray(fs["cloud"].ravel()), *want)
    for nm, w in zip(("Dx", "Dy", "Dz", "lap", "lapP"), want):
        if nm != "Dz" or dim == 3:
            assert np.array_equal(got[nm], w.reshape(F.n, k)), nm
    pts = api.nearest_points(fs["x"], fs["y"], fs["z"], cs["x"], cs["y"], cs["z"], dim)
    for rows_from, only in ((F.nb, 0), (0, 1), (0, 0)):
        got = api.transfer_weights(fs["x"], fs["y"], fs["z"], fs["btag"], pts, rows_from, only, cs["x"], cs["y"],
                                   cs["z"], cs["cloud"], dim, phs, poly)
        want = np.zeros(F.n * k)
        O.lib(True).orc_transfer_weights(F.n, fs["x"], fs["y"], fs["z"], fs["btag"], pts, rows_from, only, C.n, k, dim,
                                         phs, poly, cs["x"], cs["y"], cs["z"],
                                         np.ascontiguousarray(cs["cloud"].ravel()), want)
        assert np.array_equal(got, want.reshape(F.n, k)), (rows_from, only)
