import glob
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")


def golden_files():
    return sorted(glob.glob(os.path.join(GOLDEN, "ka_*.npz")))


def load_golden(path):
    d = np.load(path)
    out = {k: d[k] for k in d.files}
    out["name"] = os.path.basename(path)[3:-4]
    return out


def shifted_configuration(n, box, seed):
    """A KA configuration in a box, and the same with half of the particles moved
    by whole box lengths; every coordinate a multiple of 2^-12, so that both
    hold the same separations exactly, in float32 too."""
    rng = np.random.default_rng(seed)
    box = np.array(box, np.float32)
    assert np.array_equal(box * 4096, np.rint(box * 4096))
    m = np.ceil(box / np.cbrt(np.prod(box) / n)).astype(int)
    sites = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3)
    sites = sites[np.sort(rng.permutation(len(sites))[:n])]
    x = (sites + 0.5) * (box / m) - box / 2 + 0.06 * rng.standard_normal((n, 3))
    x -= box * np.rint(x / box)
    pos4 = np.zeros((n, 4), np.float32)
    pos4[:, :3] = np.rint(x * 4096) / 4096
    types = (rng.random(n) < 0.2).astype(np.int32)
    pos4[:, 3] = types.view(np.float32)
    out = pos4.copy()
    k = rng.integers(-2, 3, (n, 3)) * (rng.random((n, 1)) < 0.5)
    out[:, :3] += (k * box).astype(np.float32)
    return box, types, pos4, out, k.astype(np.int32)


@pytest.fixture(scope="session")
def oracle():
    from oracle import oracle as O
    O.build()
    return O
