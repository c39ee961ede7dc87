"""Initialisation and output of structured boxes in node order: a periodic box is initialised at one parity
only, and must hold the populations of a box whose mask (all fluid) keeps both passes; fields of
ragged boxes come back as they went in."""
import numpy as np
import pytest

from virtualfluids_b200 import Box

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["f64", "f32", "f16"])
@pytest.mark.parametrize("shape", [(2, 2, 2), (5, 3, 2), (33, 4, 3), (129, 3, 5)], ids=lambda s: "x".join(map(str, s)))
def test_one_pass_initialisation_equals_both(cuda, storage, shape):
    rng = np.random.default_rng(3)
    n = shape[0] * shape[1] * shape[2]
    f = [rng.uniform(-a, a, n) for a in (1e-2, 0.03, 0.03, 0.03)]
    boxes = [Box(*shape, 1.9, storage=storage, mask=m) for m in (None, np.ones(n, dtype=np.uint8))]
    for b in boxes:
        b.init(*f)
    (p, even_p), (q, even_q) = (b.read_populations() for b in boxes)
    assert np.array_equal(p, q) and even_p and even_q
    got = [b.fields() for b in boxes]
    for k, want in zip(("rho", "vx", "vy", "vz"), f):
        assert np.array_equal(got[0][k], got[1][k])
        # 27 stored values summed: each rounded to the storage's spacing at |(f - w) / w| < 0.25
        eps = {"f64": 2.0 ** -55, "f32": 2.0 ** -26, "f16": 2.0 ** -12}[storage]
        assert np.abs(got[0][k] - want).max() <= 27 * eps
