"""The list collision with two entries per thread (large levels with walls, FP32 arithmetic) on the GPU, with the
entry count on either side of the size from which two are taken and not a multiple of the warp's 64:
the populations of the list kernel with one entry (no slot table) in every storage, and in FP32 the
fields of the structured-box form of the same level with one node per thread, bit for bit."""
import numpy as np
import pytest

from virtualfluids_b200 import BoundaryConditionFactory as BCF
from virtualfluids_b200 import Box, ListGrid, Parameter, Simulation
from virtualfluids_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(57, 54, 49), (57, 54, 50)], ids=["below", "above"])
def test_two_list_entries_per_thread_equal_the_box(cuda, shape):
    assert (shape[0] * shape[1] * shape[2] >= 148 * 4 * 256) == (shape[2] == 50)
    grid = ListGrid(*shape)
    for side in ("PX", "MX", "PY", "MY", "MZ"):
        grid.add_side(side, "noslip")
    grid.add_side("PZ", "velocity", velocity=(0.05, 0.02, 0.0))
    bcf = BCF()
    bcf.set_no_slip_boundary_condition(BCF.NoSlipBC.NoSlipInterpolatedCompressible)
    bcf.set_velocity_boundary_condition(BCF.VelocityBC.VelocityInterpolatedCompressible)
    p = Parameter()
    p.set_viscosity_lb(0.01)
    p.configure_main_kernel("K17CompressibleNavierStokes")
    p.storage, p.arith = N.STORAGE_F32, N.ARITH_FAST
    rng = np.random.default_rng(8)
    n = grid.number_of_nodes
    f = [rng.uniform(-a, a, n) * (grid.geo == N.GEO_FLUID) for a in (1e-3, 0.02, 0.02, 0.02)]
    sim = Simulation(p, grid, bcf)
    sim.init(*f)
    box = Box.from_grid(grid, p.omega, bcf, storage="f32")
    box.set_kernel_variant("direct")
    f0 = grid.first_node
    box.init(*(np.ascontiguousarray(a[f0:f0 + box.n]) for a in f))
    sim.run(5)
    box.step(5)
    got, want = sim.macroscopic(), box.fields()
    for k, kb in (("rho", "rho"), ("vx", "vx"), ("vy", "vy"), ("vz", "vz")):
        assert np.array_equal(got[k][f0:f0 + box.n].astype(np.float32), want[kb])


@pytest.mark.parametrize("storage", [N.STORAGE_F32, N.STORAGE_F16, N.STORAGE_BF16, N.STORAGE_E3M12],
                         ids=["f32", "f16", "bf16", "e3m12"])
@pytest.mark.parametrize("shape", [(57, 54, 50), (61, 59, 53)], ids=lambda s: "x".join(map(str, s)))
def test_two_list_entries_per_thread_equal_one(cuda, storage, shape):
    grid = ListGrid(*shape)
    for side in ("PX", "MX", "PY", "MY", "MZ", "PZ"):
        grid.add_side(side, "noslip")
    assert grid.fluid.size >= 151552 and grid.fluid.size % 64
    bcf = BCF()
    bcf.set_no_slip_boundary_condition(BCF.NoSlipBC.NoSlipBounceBack)
    p = Parameter()
    p.set_viscosity_lb(0.01)
    p.configure_main_kernel("K17CompressibleNavierStokes")
    p.storage, p.arith = storage, N.ARITH_FAST
    rng = np.random.default_rng(9)
    f = [rng.uniform(-a, a, grid.number_of_nodes) * (grid.geo == N.GEO_FLUID) for a in (1e-3, 0.02, 0.02, 0.02)]
    out = []
    for tables in (0, 1):
        sim = Simulation(p, grid, bcf, neighbor_tables=tables)
        sim.init(*f)
        sim.run(5)
        out.append(sim.populations())
        sim.close()
    assert np.array_equal(out[0], out[1])
