"""The pool's host side on a CUDA runtime without a device (fake_cudart.cpp): which collision kernel a step
launches, on which grid, and what happens when a query fails. Domains of 4 GB a plane are address
space only."""
import ctypes as C

import pytest

from virtualfluids_b200 import _native as N
from virtualfluids_b200.pool import Pool

SMS, OCC_NARROW, OCC_WIDE = 148, 5, 3           # of the fake runtime


class FakePool:
    """The C ABI's pool on the fake runtime."""

    def __init__(self, lib, storage, gigabytes):
        self.lib, self.h = lib, C.c_void_p()
        d = N.PoolDesc(storage, N.ARITH_FAST, int(gigabytes * 2 ** 30), 16)
        assert lib.vfb_pool_create(C.byref(d), C.byref(self.h)) == 0

    def add(self, shape):
        i, any_pointer = C.c_uint32(), C.c_void_p(4096)
        assert self.lib.vfb_pool_add_domain(self.h, C.byref(Pool.desc(shape, 1.8)), None, C.byref(i)) == 0
        assert self.lib.vfb_pool_init_domain(self.h, i, *[any_pointer] * 4, 0, None) == 0
        return i

    def remove(self, i):
        assert self.lib.vfb_pool_remove_domain(self.h, i) == 0

    def set_launch(self, threads, nodes_per_thread, blocks_per_sm):
        assert self.lib.vfb_pool_set_launch(self.h, threads, nodes_per_thread, blocks_per_sm, 0) == 0

    def step(self):
        return self.lib.vfb_pool_step(self.h, 1, None)

    def last_launch(self):
        """(32-bit slot offsets, grid, threads) of the last launch, a collision."""
        grid, block = C.c_uint(), C.c_uint()
        name = self.lib.fake_launch(self.lib.fake_launches() - 1, C.byref(grid), C.byref(block)).decode()
        assert "k17_pool_kernel" in name
        return "Lb1EEEv" in name, grid.value, block.value

    def close(self):
        self.lib.vfb_pool_destroy(self.h)


def test_a_failed_change_of_kernel_is_reported_and_made_good(fake_lib):
    p = FakePool(fake_lib, N.STORAGE_F32, 120)
    p.set_launch(128, 8, 0)
    p.add((64, 64, 64))
    assert p.step() == 0 and p.last_launch() == (True, SMS * OCC_NARROW, 128)
    big = p.add((1024, 1024, 1024))             # planes of 4 GB: 64-bit slot offsets
    fake_lib.fake_fail_occupancy(1)
    before = fake_lib.fake_launches()
    assert p.step() != 0 and fake_lib.fake_launches() == before
    assert p.step() == 0 and p.last_launch() == (False, SMS * OCC_WIDE, 128)
    p.remove(big)
    assert p.step() == 0 and p.last_launch() == (True, SMS * OCC_NARROW, 128)
    p.close()


def test_a_work_list_without_memory_is_formed_again(fake_lib):
    p = FakePool(fake_lib, N.STORAGE_F32, 1)
    p.add((64, 64, 64))
    assert p.step() == 0
    for _ in range(8):
        p.add((64, 64, 64))                     # more items than the list holds
    fake_lib.fake_fail_malloc(1)
    before = fake_lib.fake_launches()
    assert p.step() != 0 and fake_lib.fake_launches() == before
    assert p.step() == 0 and p.last_launch() == (True, 9 * 64 ** 3 // (128 * 8), 128)
    p.close()


@pytest.mark.parametrize("storage,width", [(N.STORAGE_F64, 1), (N.STORAGE_F32, 2), (N.STORAGE_F16, 2)], ids=["f64", "f32", "f16"])
@pytest.mark.parametrize("nodes_per_thread", [1, 2, 3, 8])
def test_items_hold_whole_multiples_of_a_threads_nodes(fake_lib, storage, width, nodes_per_thread):
    p = FakePool(fake_lib, storage, 1)
    p.set_launch(64, nodes_per_thread, -1)      # one block per item
    p.add((40, 30, 20))
    assert p.step() == 0
    per_item = 64 * -(-nodes_per_thread // width) * width
    assert p.last_launch()[1:] == (-(-24000 // per_item), 64)
    p.close()
