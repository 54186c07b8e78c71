"""set_X / get_X of a batch: meshes small and large, page-locked and pageable
arrays, one host thread and several."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from egg_b200 import configs

pytestmark = pytest.mark.gpu

# 32768 reals (128 x 128 nodes) are worth a DMA of their own; 4 MiB of staged
# reals a host thread
SIDES = {"small": [5, 9, 3, 17] * 40, "mixed": [5, 129, 9, 127, 128, 3, 300], "threads": [513, 9, 700, 129, 513, 7]}


def _batch(gpu, sides):
    gs = {n: configs.unit_square(n, frac=0.2, seed=n) for n in set(sides)}
    ws = {n: (g.wire(compact=True), g.structured(), g.X_flat()) for n, g in gs.items()}
    return gpu.CppBatchSweepSession([ws[n] for n in sides])


def _array(n, seed, pinned):
    x = np.random.default_rng(seed).uniform(-1.0, 1.0, 2 * n * n)
    return torch.from_numpy(x).pin_memory().numpy() if pinned else x


@pytest.mark.parametrize("pinned", ["none", "all", "every other", "last"])
@pytest.mark.parametrize("name", list(SIDES))
def test_positions_come_back(gpu, name, pinned):
    sides = SIDES[name]
    b = _batch(gpu, sides)
    for seed in (0, 1000):  # twice: the staging is in use again
        pin = [{"none": False, "all": True, "every other": m % 2 == 0, "last": m == len(sides) - 1}[pinned]
               for m in range(len(sides))]
        X = [_array(n, seed + m, p) for m, (n, p) in enumerate(zip(sides, pin))]
        b.set_X(X)
        for x, y in zip(X, b.get_X()):
            np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("name", list(SIDES))
def test_arrays_own_their_memory(gpu, name):
    """A mesh that a caller keeps holds nothing of the others."""
    b = _batch(gpu, SIDES[name])
    X = b.get_X()
    for x in X:
        assert x.flags.owndata and x.base is None and x.flags.writeable
    keep = X[1].copy()
    X[0][:] = 7.0
    np.testing.assert_array_equal(X[1], keep)
    X[1].resize(2, refcheck=False)
    np.testing.assert_array_equal(b.get_X()[1], keep)
