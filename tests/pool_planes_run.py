"""Run by tests/test_gpu_pool_planes.py in a process of its own (a process loads one build of the library). Steps
a pool whose work list gains and loses a domain with planes above 1 MB; prints one JSON line with a
hash of every domain's fields after each phase."""
import hashlib
import json
import sys
from pathlib import Path

import numpy as np

sys.path.insert(0, str(Path(__file__).resolve().parent.parent))

from virtualfluids_b200 import Pool  # noqa: E402
from virtualfluids_b200 import _native as N  # noqa: E402

BIG = (85, 84, 83)      # planes of 1.2 MB in 16 bits


def fields(shape, seed):
    rng = np.random.default_rng(seed)
    n = shape[0] * shape[1] * shape[2]
    return [rng.uniform(-a, a, n) for a in (1e-2, 0.03, 0.03, 0.03)]


def main():
    import torch
    out = {"checked": N.lib().vfb_bounds_checked()}
    for storage in ("f32", "f16", "bf16", "e3m12", "f64"):
        for blocks_per_sm in (-1, 0):
            pool = Pool(500 << 20, storage=storage, max_domains=8)
            pool.set_launch(128, 8, blocks_per_sm)
            stream = torch.cuda.Stream()
            hashes = []

            def add(shape, seed, **kw):
                i = pool.add(shape, 1.9, **kw)
                pool.init(i, *fields(shape, seed), stream=stream)
                return i

            def phase():
                pool.step(19, stream=stream)        # a graph of 16 steps and three launched ones
                for i in sorted(pool.domains):
                    h = hashlib.sha256()
                    for a in pool.fields(i, stream=stream):
                        h.update(np.ascontiguousarray(a).tobytes())
                    hashes.append(h.hexdigest())

            rng = np.random.default_rng(2)
            add((33, 17, 9), 1)
            add((40, 30, 20), 2, periodic=(True, False, False), forces=(1e-5, 0.0, 0.0))
            add((32, 31, 30), 3, mask=(rng.random(32 * 31 * 30) < 0.7).astype(np.uint8))
            phase()
            big = add(BIG, 4, forces=(0.0, 1e-5, 0.0))
            phase()
            pool.remove(big)
            phase()
            out[f"{storage} {blocks_per_sm}"] = hashes
            pool.close()
    print(json.dumps(out))


if __name__ == "__main__":
    main()
