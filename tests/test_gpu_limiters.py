"""Quadric limiters far from the default 0.01 on the GPU: infinite, very large (the limiter is off), very
small. The exact arithmetic computes the oracle's bits with each of them."""
import numpy as np
import pytest

from virtualfluids_b200 import BoundaryConditionFactory as BCF
from virtualfluids_b200 import ListGrid, Parameter, Simulation
from virtualfluids_b200 import _native as N

pytestmark = pytest.mark.gpu

LIMITERS = [(np.inf, np.inf, np.inf), (1e300, 0.01, 1e-300), (1e45, 1e45, 1e45), (0.01, np.inf, 1e40)]


def _fields(n, seed):
    rng = np.random.default_rng(seed)
    f = [rng.uniform(-a, a, n) for a in (1e-2, 0.03, 0.03, 0.03)]
    for v in f:
        v[0] = 0.0
    return f


@pytest.mark.parametrize("limiters", LIMITERS, ids=str)
def test_exact_arithmetic_with_any_limiter_matches_the_oracle(oracle, cuda, limiters):
    grid = ListGrid(9, 7, 5, periodic=(True, True, True))
    p = Parameter()
    p.set_viscosity_lb(0.01)
    p.configure_main_kernel("K17CompressibleNavierStokes")
    p.set_quadric_limiters(*limiters)
    p.storage, p.arith = N.STORAGE_F64, N.ARITH_EXACT
    f = _fields(grid.number_of_nodes, 4)
    sim = Simulation(p, grid, BCF())
    sim.init(*f)
    sim.run(6)
    orc = oracle.OracleLevel(grid, omega=p.omega, lim=limiters)
    orc.init(*f)
    orc.run(6)
    assert np.isfinite(orc.f).all() and np.array_equal(sim.populations(), orc.f)
