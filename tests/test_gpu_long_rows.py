"""Boxes with rows of 65536 nodes and more on the GPU, where the box kernels' index arithmetic is the
hardware division (csrc/kernels.cuh box_slots): the collision against the list kernel of the same
level, bit for bit, and fields that come back as they went in."""
import numpy as np
import pytest

from virtualfluids_b200 import BoundaryConditionFactory as BCF
from virtualfluids_b200 import Box, ListGrid, Parameter, Simulation
from virtualfluids_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["direct", "pairs"])
@pytest.mark.parametrize("shape", [(65535, 2, 2), (65536, 3, 2), (70001, 2, 3)], ids=lambda s: "x".join(map(str, s)))
def test_long_rows_equal_the_list_kernel(cuda, shape, variant):
    grid = ListGrid(*shape, periodic=(True, True, True))
    p = Parameter()
    p.set_viscosity_lb(0.01)
    p.configure_main_kernel("K17CompressibleNavierStokes")
    p.storage, p.arith = N.STORAGE_F32, N.ARITH_FAST
    rng = np.random.default_rng(8)
    f = [rng.uniform(-a, a, grid.number_of_nodes) for a in (1e-3, 0.02, 0.02, 0.02)]
    for v in f:
        v[0] = 0.0
    sim = Simulation(p, grid, BCF(), neighbor_tables=0)
    sim.init(*f)
    box = Box(*shape, p.omega, storage="f32")
    box.set_kernel_variant(variant)
    f0 = grid.first_node
    box.init(*(np.ascontiguousarray(a[f0:f0 + box.n]) for a in f))
    for k, v in zip(("rho", "vx", "vy", "vz"), f):
        # 27 stored values summed: each rounded to 2^-26 at |(f - w) / w| < 0.25
        assert np.abs(box.fields()[k] - v[f0:f0 + box.n]).max() <= 27 * 2.0 ** -26
    sim.run(5)
    box.step(5)
    got, want = sim.macroscopic(), box.fields()
    for k in ("rho", "vx", "vy", "vz"):
        assert np.array_equal(got[k][f0:f0 + box.n].astype(np.float32), want[k])
