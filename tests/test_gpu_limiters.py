"""Quadric limiters far from the default 0.01 on the GPU: infinite, very large (the limiter is off), very
small. The exact arithmetic computes the oracle's bits with each of them, and the FMA arithmetic one result
for all that are off."""
import numpy as np
import pytest

from virtualfluids_b200 import BoundaryConditionFactory as BCF
from virtualfluids_b200 import Box, ListGrid, Parameter, Simulation
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


@pytest.mark.parametrize("storage,arith", [("f64", "fast"), ("f32", "fast"), ("f32", "exact"), ("f16", "fast")])
def test_limiters_that_are_off_give_one_result(cuda, storage, arith):
    shape, n = (33, 9, 8), 33 * 9 * 8
    f = _fields(n, 5)
    out = []
    for q in (2.0 ** 100, 1e38, np.inf):
        b = Box(*shape, 1.9, storage=storage, arith=arith, quadric_limiters=(q, q, q))
        b.init(*f)
        b.step(5)
        assert all(np.isfinite(v).all() for v in b.fields().values())
        out.append(b.read_populations()[0])
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("storage", ["f64", "f32"])
def test_infinite_limiters_fma_against_exact(cuda, storage):
    shape, n = (33, 9, 8), 33 * 9 * 8
    f = _fields(n, 6)
    got = []
    for arith in ("exact", "fast"):
        b = Box(*shape, 1.9, storage=storage, arith=arith, quadric_limiters=(np.inf, 0.01, np.inf))
        b.init(*f)
        b.step(5)
        got.append(b.fields())
    # five collisions of some 500 operations on moments of O(0.1), each rounded to 2^-53 or 2^-24
    eps = 5 * 500 * 0.1 * 2.0 ** (-53 if storage == "f64" else -24)
    for k in ("rho", "vx", "vy", "vz"):
        assert np.abs(got[0][k] - got[1][k]).max() <= eps
