"""The 2D interior kernels at the edges of their tiles, in every tile variant,
and the DOFs that the mixed path relaxes in fp64."""

from __future__ import annotations

import numpy as np
import pytest

from egg_b200 import configs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _box(shape, frac, seed):
    """One block of unequal node counts, spacing 1 along both axes."""
    ids = np.arange(int(np.prod(shape)), dtype=np.int64).reshape(shape)
    X = np.stack(np.meshgrid(*[np.arange(n, dtype=float) for n in shape], indexing="ij"), axis=-1).reshape(-1, 2)
    free = np.zeros(shape, dtype=bool)
    free[1:-1, 1:-1] = True
    free = free.reshape(-1)
    X[free] += np.random.default_rng(seed).uniform(-frac, frac, (int(free.sum()), 2))
    return configs.Grid("box", 2, [ids], X, free)


def _oracle(g, phase, delta):
    return oracle.run(g.X, oracle.patches_for(g.blocks, g.free), oracle.stencil_for(g.blocks), 1, phase=phase,
                      delta=delta, omega=0.9)


@pytest.mark.parametrize("phase,delta", [("barrier", 0.0), ("shape_size", 0.0), ("untangle", 0.1)])
@pytest.mark.parametrize("shape", [(3, 3), (10, 18), (11, 19), (19, 35)], ids=str)
def test_tile_edges_match_oracle(gpu, shape, phase, delta):
    """Well-shaped cells, spacing 1: fp64 to rounding (1e-12 of the spacing),
    mixed within the 1e-5 that its first sweep promises."""
    g = _box(shape, 0.15, 4)
    Xo, Eo, _ = _oracle(g, phase, delta)
    for precision, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
        for variant in range(5):
            s = gpu.CppStructuredSweepSession(g.wire(), g.structured(), g.X_flat(), precision=precision)
            s.set_variant(variant)
            E, _ = s.run(1, phase=phase, delta=delta, omega=0.9)
            assert np.abs(s.get_X().reshape(-1, 2) - Xo).max() <= tol
            np.testing.assert_allclose(E, Eo, rtol=1e-12 if precision == "fp64" else 1e-5)


@pytest.mark.parametrize("phase,delta", [("barrier", 0.0), ("untangle", 0.05)])
def test_mixed_dofs_next_to_bad_cells_relax_in_fp64(gpu, phase, delta):
    """+-0.4 noise on a 35 x 50 block: inverted and badly shaped cells, some
    warps with none, one or several of their DOFs.  A DOF with a clearly bad
    sample (sine below 0.07, or inverted) takes 16 lanes in fp64; where no
    sample around it is closer to degenerate than sine 1e-2, its H is
    conditioned to 1e4, so sums in another order agree to 1e-11 of the
    spacing."""
    g = _box((35, 50), 0.4, 9)
    ids = np.asarray(g.blocks[0])
    Xb = g.X[ids]
    q = []
    for b in range(4):
        i, j = b >> 1, b & 1

        def at(u, v):
            return Xb[u:34 + u, v:49 + v]

        e0 = (at(1 - i, j) - at(i, j)) * (-1 if i else 1)
        e1 = (at(i, 1 - j) - at(i, j)) * (-1 if j else 1)
        q.append((e0[..., 0] * e1[..., 1] - e0[..., 1] * e1[..., 0]) /
                 np.sqrt((e0 ** 2).sum(-1) * (e1 ** 2).sum(-1)))
    q = np.stack(q, -1)
    bad, near = (q < 0.07).any(-1), (np.abs(q) < 1e-2).any(-1)
    touch = lambda m: m[:-1, :-1] | m[:-1, 1:] | m[1:, :-1] | m[1:, 1:]  # noqa: E731
    pick = ids[1:-1, 1:-1][touch(bad) & ~touch(near)]
    assert pick.size > 50
    Xo, _, _ = _oracle(g, phase, delta)
    for variant in range(5):
        s = gpu.CppStructuredSweepSession(g.wire(), g.structured(), g.X_flat(), precision="mixed")
        s.set_variant(variant)
        s.run(1, phase=phase, delta=delta, omega=0.9)
        assert np.abs(s.get_X().reshape(-1, 2) - Xo)[pick].max() <= 1e-11
