"""The two-node kernels (packed FP32x2 arithmetic) on the GPU: the same bits as one node per thread, at
sizes around the 64 nodes of a warp, with walls, and on either side of the size from which a box
takes two nodes per thread by itself."""
import numpy as np
import pytest

from virtualfluids_b200 import Box

pytestmark = pytest.mark.gpu

SHAPES = [(2, 2, 2), (3, 5, 7), (7, 3, 3), (8, 4, 2), (13, 5, 2), (31, 3, 3), (65, 4, 3), (33, 17, 9)]


def _state(shape, seed):
    rng = np.random.default_rng(seed)
    n = shape[0] * shape[1] * shape[2]
    return [rng.uniform(-a, a, n) for a in (1e-2, 0.03, 0.03, 0.03)]


def _run(shape, storage, variant, steps, periodic=(True, True, True)):
    nx, ny, nz = shape
    mask = None
    if not all(periodic):
        z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
        wall = np.zeros(x.shape, dtype=bool)
        for c, n, p in ((x, nx, periodic[0]), (y, ny, periodic[1]), (z, nz, periodic[2])):
            if not p:
                wall |= (c == 0) | (c == n - 1)
        mask = (~wall).astype(np.uint8).reshape(-1)
    b = Box(nx, ny, nz, 1.9, periodic=periodic, storage=storage, forces=(1e-5, 0.0, -2e-5), mask=mask)
    b.set_kernel_variant(variant)
    # the slots that belong to solid nodes alone are never written: the same in every box
    b.write_populations(np.zeros_like(b.read_populations()[0]))
    b.init(*_state(shape, 5))
    energy = np.zeros((steps, 2))
    b.step(steps, energy=energy)
    pops, even = b.read_populations()
    return pops, even, energy


@pytest.mark.parametrize("storage", ["f32", "f16", "bf16", "e3m12"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_two_nodes_per_thread_give_the_bits_of_one(cuda, storage, shape):
    for periodic in ((True, True, True), (True, False, False)):
        if not all(periodic) and min(shape[1:]) < 3:
            continue
        one, two = (_run(shape, storage, v, 5, periodic) for v in ("direct", "pairs"))
        assert np.array_equal(one[0], two[0]) and one[1] == two[1]
        # the FP64 sums run in another order: n terms of O(1), each sum rounded to 2^-53
        assert np.allclose(one[2], two[2], rtol=1e-12, atol=0)


# on either side of 200 000 (FP32, E3M12) and 1 600 000 nodes (FP16, BF16); tests/test_dispatch_host.py reads
# which kernel a step launches there
@pytest.mark.parametrize("storage,shape", [("f32", (57, 59, 59)), ("f32", (58, 59, 59)), ("e3m12", (58, 59, 59)),
                                           ("f16", (116, 117, 117)), ("f16", (117, 117, 117)), ("bf16", (117, 117, 117))])
def test_the_choice_by_size_changes_no_bit(cuda, storage, shape):
    a, b, c = (_run(shape, storage, v, 3) for v in ("auto", "direct", "pairs"))
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[0], c[0])
