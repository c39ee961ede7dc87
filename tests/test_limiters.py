"""Quadric limiters far above the default 0.01 (the limiter is off; any double is accepted) in the FMA form
of the collision: each limited moment comes out as in the exact form, for limiters up to infinity."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = tmp_path_factory.mktemp("limiter") / "check.so"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-shared",
                    "-gencode", "arch=compute_100a,code=sm_100a", "-Xcompiler", "-fPIC,-ffp-contract=off",
                    f"-I{ROOT / 'virtualfluids_b200' / 'csrc'}", str(ROOT / "tests" / "limiter_check.cu"), "-o", str(so)],
                   check=True)
    lib = ctypes.CDLL(str(so))
    lib.limiter_difference.argtypes = [ctypes.c_int] + 3 * [ctypes.c_double] + [ctypes.c_int]
    lib.limiter_difference.restype = ctypes.c_double
    return lib


@pytest.mark.parametrize("real_bytes", [8, 4], ids=["f64", "f32"])
@pytest.mark.parametrize("limiters", [(0.01, 0.01, 0.01), (1e6, 1e6, 1e6), (1e29, 1e31, 1e38), (1e45, 1e45, 1e45),
                                      (1e300, 0.01, 0.01), (np.inf, np.inf, np.inf), (0.01, np.inf, 1e-20)], ids=str)
def test_fma_form_equals_the_exact_form_for_large_limiters(check, real_bytes, limiters):
    # populations and moments of O(0.1) (27 values below 0.02), some 500 operations, each rounded to 2^-53 or 2^-24
    assert check.limiter_difference(real_bytes, *limiters, 2000) <= 0.1 * 500 * 2.0 ** (-53 if real_bytes == 8 else -24)
