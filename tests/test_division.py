"""The exact collision's division (csrc/k17.cuh) against the IEEE division, bit for bit.

refine_rcp and refine_div, the part without a branch: for every seed within 2^-18 of the reciprocal,
with fractions at both ends of a binade (the all-ones divisor, where the last refinement alone gives
the wrong neighbour; powers of two) and over wide exponents. rcp_rounded and limited, the whole: for any
operands (both signs, zeros, subnormals, infinities, NaN, exponents around the limits of the range that the
first part serves) and any limiters, on the host and on the device with the hardware's approximation. The
collision's own 1 / rho has no branch: where rho is 0, infinite or huge, its populations must be those with
the IEEE reciprocal all the same."""
import ctypes
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = tmp_path_factory.mktemp("division") / "check.so"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-shared",
                    "-gencode", "arch=compute_100a,code=sm_100a", "-fmad=false", "-Xcompiler", "-fPIC,-ffp-contract=off", f"-I{ROOT / 'virtualfluids_b200' / 'csrc'}",
                    str(ROOT / "tests" / "division_check.cu"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.division_mismatches.argtypes = [ctypes.c_long, ctypes.c_uint64, ctypes.c_int]
    lib.division_mismatches.restype = ctypes.c_long
    for f in (lib.whole_mismatches, lib.device_mismatches):
        f.argtypes, f.restype = [ctypes.c_long, ctypes.c_int], ctypes.c_long
    return lib


@pytest.mark.parametrize("exponents", [1, 40, 400])
def test_rounded_division_is_the_ieee_division(check, exponents):
    assert check.division_mismatches(1_000_000, 0x9E3779B97F4A7C15 + exponents, exponents) == 0


@pytest.mark.parametrize("wide", [0, 1], ids=["in_range", "any"])
def test_whole_division_is_the_ieee_division(check, wide):
    assert check.whole_mismatches(300_000, wide) == 0


def test_populations_where_the_density_has_no_reciprocal(check):
    check.density_mismatches.argtypes, check.density_mismatches.restype = [ctypes.c_long], ctypes.c_long
    assert check.density_mismatches(40_000) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("wide", [0, 1], ids=["in_range", "any"])
def test_device_division_is_the_ieee_division(cuda, check, wide):
    assert check.device_mismatches(50_000_000, wide) == 0
