"""The exact collision's branch-free division (csrc/k17.cuh refine_rcp, refine_div) against the host's
IEEE division: rounded reciprocals and quotients must be the same bits for every seed within 2^-18
of the reciprocal, with fractions at both ends of a binade (the all-ones divisor, where the last
refinement alone gives the wrong neighbour; powers of two) and over wide exponents."""
import ctypes
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    so = tmp_path_factory.mktemp("division") / "check.so"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-shared",
                    "-Xcompiler", "-fPIC,-ffp-contract=off", f"-I{ROOT / 'virtualfluids_b200' / 'csrc'}",
                    str(ROOT / "tests" / "division_check.cu"), "-o", str(so)], check=True)
    lib = ctypes.CDLL(str(so))
    lib.division_mismatches.argtypes = [ctypes.c_long, ctypes.c_uint64, ctypes.c_int]
    lib.division_mismatches.restype = ctypes.c_long
    return lib


@pytest.mark.parametrize("exponents", [1, 40, 400])
def test_rounded_division_is_the_ieee_division(check, exponents):
    assert check.division_mismatches(1_000_000, 0x9E3779B97F4A7C15 + exponents, exponents) == 0
