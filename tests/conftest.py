import ctypes
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200)")


def pytest_collection_modifyitems(items):
    # GPU tests against the reference's own kernels and grid generator fail where those are not built
    # (oracle/_ref); they run last then, so that a run which stops at the first failure has run the others
    if not (ROOT / "oracle" / "_ref" / "libvfref_gpu64.so").exists():
        def pinned(item):
            return any(w in item.nodeid for w in ("test_gpu_gridgen.py", "test_gpu_reference_kernels.py",
                                                  "matches_reference_kernel", "match_reference_kernels"))
        items.sort(key=pinned)


@pytest.fixture(scope="session")
def oracle():
    from oracle import pyoracle
    pyoracle.lib()
    return pyoracle


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("a CUDA device is required for gpu-marked tests")
    return torch.device("cuda:0")


@pytest.fixture(scope="session")
def fake_lib(tmp_path_factory):
    """The library on a CUDA runtime without a device (fake_cudart.cpp)."""
    from virtualfluids_b200 import build as vbuild
    vbuild.build()
    out = tmp_path_factory.mktemp("fake") / "libvfb_fake.so"
    # -Bsymbolic: the objects' calls go to the fake runtime whatever else the process has loaded
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I/usr/local/cuda/include",
                    str(ROOT / "tests" / "fake_cudart.cpp"), *map(str, sorted(vbuild.BUILD.glob("*.o"))),
                    "-Wl,-Bsymbolic", "-Wl,-z,defs", "-ldl", "-lrt", "-lpthread", "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    lib.fake_launch.restype = ctypes.c_char_p
    return lib
