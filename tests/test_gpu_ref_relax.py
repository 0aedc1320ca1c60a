"""Reference-mode relaxation and cycle for every parity of the sweep count:
several sweeps in one call give the bits of as many calls of one sweep (each
re-pinning p and taking the residual, whose last value is kept), and the
cycle, which takes a relaxation's last residual and the interior residual in
one pass, the bits of the routines called one by one."""
import numpy as np
import pytest

import multigrid_meshless_b200 as mgm
from multigrid_meshless_b200 import api, clouds

pytestmark = pytest.mark.gpu

SHAPES = {"cavity": (clouds.cavity_hierarchy, (36, 3), 20, 3), "cube": (clouds.cube_hierarchy, (12, 2), 30, 2)}


@pytest.fixture(params=list(SHAPES))
def mg(request):
    fn, a, k, poly = SHAPES[request.param]
    cl = fn(*a)
    m = api.Multigrid(cl, [k] * len(cl), [poly] * len(cl), reference_transfer=True)
    yield m
    m.close()


def _load(m, seed):
    rng = np.random.default_rng(seed)
    for l in range(m.nl):
        for nm in ("p", "res", "source"):
            m.set_field(nm, rng.standard_normal(m.n(l)), l)


def _state(m):
    return [m.get_field(nm, l) for nm in ("p", "res") for l in range(m.nl)]


@pytest.mark.parametrize("sweeps", [0, 1, 2, 3, 4])
def test_sweep_counts(mg, sweeps):
    out = []
    for together in (True, False):
        _load(mg, 3)
        mg.set_flow(Re=100.0, courant=0.5, omega=0.3, num_relax=sweeps if together else 1, num_vcycles=2)
        for l in range(mg.nl):
            for _ in range(1 if together else sweeps):
                mg.ref_routine(l, "relaxation")
        out.append(_state(mg))
    assert all(np.array_equal(a, b) for a, b in zip(*out))


@pytest.mark.parametrize("sweeps", [0, 1, 2, 3])
def test_cycle_is_its_routines(mg, sweeps):
    mg.set_flow(Re=100.0, courant=0.5, omega=0.3, num_relax=sweeps, num_vcycles=2)
    out = []
    for by_routine in (False, True):
        _load(mg, 4)
        if by_routine:
            for _ in range(2):
                for l in range(mg.nl):
                    mg.ref_routine(l, "relaxation")
                    mg.ref_routine(l, "residuals")
                    if l != mg.nl - 1:
                        mg.ref_routine(l, "restrict")
                for l in range(mg.nl - 1, 0, -1):
                    mg.ref_routine(l - 1, "prolongate")
                    if l != 1:
                        mg.ref_routine(l - 1, "relaxation")
        else:
            mg.poisson(mgm.MODE_REFERENCE)
        out.append(_state(mg))
    assert all(np.array_equal(a, b) for a, b in zip(*out))
