"""The 3D interior kernel at the edges of its tiles: blocks from a single DOF
to a tile plus a remainder along every axis, in every tile variant, against the
NumPy-patch oracle."""

from __future__ import annotations

import itertools

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


def _turned_cubes(perm, flips, frac=0.15, seed=2):
    """Two 5 x 4 x 6 boxes of unit cells meeting in the plane x = 4, the second
    one's axes permuted and reversed."""
    a = np.stack(np.meshgrid(*[np.arange(n, dtype=float) for n in (5, 4, 6)], indexing="ij"), axis=-1)
    b = a + np.array([4.0, 0.0, 0.0])
    b = b.transpose(*perm, 3)[tuple(slice(None, None, -1 if f else 1) for f in flips)]
    blocks, X = configs._dedupe([a, b])
    free = ((X > 0) & (X < np.array([8.0, 3.0, 5.0]))).all(axis=1)
    X = X + np.where(free[:, None], np.random.default_rng(seed).uniform(-frac, frac, X.shape), 0.0)
    return configs.Grid("turned", 3, blocks, X, free)


@pytest.mark.parametrize("perm", list(itertools.permutations(range(3))), ids=str)
def test_lattice_dofs_of_turned_blocks_match_oracle(gpu, perm):
    """The nodes of the shared face relax over a lattice table of their own
    order, whatever way the second block is turned; a mirrored block's
    negative dets (untangle) keep such a DOF on the general path.  One sweep
    of fp64 sums in another order: 1e-12 of the spacing."""
    odd = sum(perm[i] > perm[j] for i in range(3) for j in range(i + 1, 3)) % 2
    for flips in itertools.product((0, 1), repeat=3):
        mirrored = (odd + sum(flips)) % 2 == 1
        phase, delta = ("untangle", 0.3) if mirrored else ("barrier", 0.0)
        g = _turned_cubes(perm, flips)
        Xo, Eo, _ = oracle.run3(g.X, oracle.patches_for(g.blocks, g.free, d=3), oracle.stencil_for(g.blocks, d=3), 1,
                                phase=phase, delta=delta, omega=0.8)
        for precision, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
            s = gpu.CppStructuredSweepSession(g.wire(), g.structured(), g.X_flat(), dim=3, precision=precision)
            E, _ = s.run(1, phase=phase, delta=delta, omega=0.8)
            assert np.abs(s.get_X().reshape(-1, 3) - Xo).max() <= tol
            face = np.isclose(g.X[:, 0], 4.0, atol=0.2) & g.free
            assert np.abs(s.get_X().reshape(-1, 3) - Xo)[face].max() <= 1e-12  # stored DOFs relax in fp64
