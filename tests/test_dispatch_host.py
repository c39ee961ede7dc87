"""Which collision kernel a box step launches, and with how many threads per block, on either side of the
lines of the dispatch (csrc/launch_impl.cuh pair_nodes, csrc/launch.h box_threads), on a CUDA runtime
without a device (fake_cudart.cpp)."""
import ctypes as C

import pytest

from virtualfluids_b200 import _native as N

ST = {"f64": N.STORAGE_F64, "f32": N.STORAGE_F32, "f16": N.STORAGE_F16, "bf16": N.STORAGE_BF16, "e3m12": N.STORAGE_E3M12}


def _launched(lib, shape, storage, exact=False, variant=0):
    d = N.BoxDesc()
    d.nx, d.ny, d.nz = shape
    d.periodic_x = d.periodic_y = d.periodic_z = 1
    d.storage, d.arith, d.omega = ST[storage], N.ARITH_EXACT if exact else N.ARITH_FAST, 1.8
    for i in range(3):
        d.quadric_limiters[i] = 0.01
    box = C.c_void_p()
    assert lib.vfb_box_create(C.byref(d), C.byref(box)) == 0
    assert lib.vfb_box_set_kernel_variant(box, variant) == 0
    assert lib.vfb_box_step(box, 1, None, 0, None) == 0
    grid, block = C.c_uint(), C.c_uint()
    name = lib.fake_launch(lib.fake_launches() - 1, C.byref(grid), C.byref(block)).decode()
    assert lib.vfb_box_destroy(box) == 0
    nodes = 2 if "k17_box_pair_kernel" in name else 1
    assert nodes == 2 or "k17_box_kernel" in name
    assert grid.value * block.value * nodes >= shape[0] * shape[1] * shape[2]
    return nodes, block.value


@pytest.mark.parametrize("storage,exact,line", [("f32", False, 200_000), ("e3m12", False, 200_000), ("f16", False, 1_600_000),
                                                ("bf16", False, 1_600_000), ("f64", False, None), ("f64", True, None),
                                                ("f32", True, None)])
def test_nodes_per_thread(fake_lib, storage, exact, line):
    below, at = ((1000, 199, 1), (1000, 200, 1)) if line != 1_600_000 else ((1000, 1599, 1), (1000, 1600, 1))
    below, at = ((s[0] // 2, s[1], 2) for s in (below, at))
    assert _launched(fake_lib, below, storage, exact) == (1, 128)
    assert _launched(fake_lib, at, storage, exact) == (2 if line else 1, 128)
    if line:
        assert _launched(fake_lib, at, storage, exact, variant=1) == (1, 128)
        assert _launched(fake_lib, below, storage, exact, variant=4) == (2, 128)


def test_threads_per_block(fake_lib):
    assert _launched(fake_lib, (37, 16, 16), "f32") == (1, 128)      # 148 x 64 nodes
    assert _launched(fake_lib, (37, 17, 15), "f32") == (1, 32)
