"""The 3D interior kernel at the edges of its tiles: blocks from a single DOF
to a tile plus a remainder along every axis, in every tile variant, against the
NumPy-patch oracle."""

from __future__ import annotations

import numpy as np
import pytest

from egg_b200 import configs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _box(shape, frac=0.15, seed=4):
    """One block of unequal node counts, spacing 1 along every axis."""
    ids = np.arange(int(np.prod(shape)), dtype=np.int64).reshape(shape)
    X = np.stack(np.meshgrid(*[np.arange(n, dtype=float) for n in shape], indexing="ij"), axis=-1).reshape(-1, 3)
    free = np.zeros(shape, dtype=bool)
    free[1:-1, 1:-1, 1:-1] = True
    free = free.reshape(-1)
    X[free] += np.random.default_rng(seed).uniform(-frac, frac, (int(free.sum()), 3))
    return configs.Grid("box", 3, [ids], X, free)


@pytest.mark.parametrize("phase,delta", [("barrier", 0.0), ("shape_size", 0.0), ("untangle", 0.1)])
@pytest.mark.parametrize("shape", [(3, 3, 3), (4, 5, 3), (6, 6, 10), (7, 11, 19)], ids=str)
def test_tile_edges_match_oracle(gpu, shape, phase, delta):
    """Spacing 1 and well-shaped cells: fp64 sums of 32 samples differ in
    rounding order alone (1e-12 of the spacing), and a mixed sweep stays within
    the 1e-5 of the spacing that the mixed path promises."""
    g = _box(shape)
    Xo, Eo, _ = oracle.run3(g.X, oracle.patches_for(g.blocks, g.free, d=3), oracle.stencil_for(g.blocks, d=3), 1,
                            phase=phase, delta=delta, omega=0.9)
    for precision, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
        for variant in range(5):
            s = gpu.CppStructuredSweepSession(g.wire(), g.structured(), g.X_flat(), dim=3, precision=precision)
            s.set_variant(variant)
            E, _ = s.run(1, phase=phase, delta=delta, omega=0.9)
            assert np.abs(s.get_X().reshape(-1, 3) - Xo).max() <= tol
            np.testing.assert_allclose(E, Eo, rtol=1e-12 if precision == "fp64" else 1e-5)
