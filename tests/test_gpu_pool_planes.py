"""The pool's collision with 64-bit slot offsets (planes of 4 GB and more; in the bounds-checked build of 1 MB
and more) and the change to it and back while domains come and go: the fields of every domain, bit
for bit, as the default build's 32-bit offsets give them for the same small planes."""
import json
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent


def _run(library):
    r = subprocess.run([sys.executable, str(ROOT / "tests" / "pool_planes_run.py")], capture_output=True, text=True,
                       env=dict(os.environ, VFB_LIBRARY=library), cwd=str(ROOT), timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_wide_slot_offsets_give_the_bits_of_narrow_ones(cuda):
    if not (ROOT / "virtualfluids_b200" / "libvfb_checked.so").exists():
        pytest.fail("libvfb_checked.so is missing: build it with python -m virtualfluids_b200.build --checked")
    wide, narrow = _run("checked"), _run("default")
    assert wide.pop("checked") == 1 and narrow.pop("checked") == 0
    assert wide == narrow
    for hashes in narrow.values():
        assert len(hashes) == 3 + 4 + 3
