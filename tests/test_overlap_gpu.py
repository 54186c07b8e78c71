"""Blocks that overlap share nodes that lie strictly inside one of them: the
tile kernel relaxes such a node, and its copy in the other block follows."""

from __future__ import annotations

import numpy as np
import pytest

from egg_b200 import configs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _axis(lo, hi, d):
    """Points of a block of unit cells from x = lo to hi, 7 nodes (and 6 in 3D) across."""
    return np.stack(np.meshgrid(np.arange(lo, hi + 1.0), *[np.arange(n, dtype=float) for n in (7, 6)[: d - 1]],
                                indexing="ij"), axis=-1)


def _overlapping(d, free_face, seed=3):
    """Block A from x = 0 to 8, block B from 7 to 14: B's face x = 7 lies
    strictly inside A, and A's face x = 8 strictly inside B."""
    blocks, X = configs._dedupe([_axis(0, 8, d), _axis(7, 14, d)])
    top = np.array([14.0, 6.0, 5.0][:d])
    free = ((X > 0) & (X < top)).all(axis=1)
    if not free_face:
        free &= X[:, 0] != 8
    X = X + np.where(free[:, None] & (X[:, :1] != 8), np.random.default_rng(seed).uniform(-0.2, 0.2, X.shape), 0.0)
    return configs.Grid("overlap", d, blocks, X, free)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("free_face", [False, True])
@pytest.mark.parametrize("d", [2, 3])
def test_copies_of_tile_nodes_follow_their_owner(gpu, d, free_face, precision):
    """A's nodes relax in A with the face x = 8 in place, B's behind that face
    in B; a node whose owner is not the slot that relaxes it stays with its
    owner.  Positions within 1e-12 (1e-5 mixed) of the spacing after one sweep.
    The energy counts the cells between x = 7 and 8 twice, from A's nodes and
    from B's copies of them: every report equals, bit for bit, that of a fresh
    session on the same positions, whose copies the upload has written."""
    run = oracle.run if d == 2 else oracle.run3
    g = _overlapping(d, free_face)
    Xo = g.X.copy()
    at8 = np.isclose(g.X[:, 0], 8.0) & (g.X[:, 0] == 8.0)
    left = g.free & (g.X[:, 0] < 8) & ~at8
    right = g.free & (g.X[:, 0] > 8) & ~at8
    ids_b = g.blocks[1][1:]  # from x = 8 on
    for ids, free in ((g.blocks[0], left), (ids_b, right)):
        X1, _, _ = run(g.X, oracle.patches_for([ids], free, d=d), oracle.stencil_for([ids], d=d), 1, omega=0.9)
        Xo[free] = X1[free]
    tol = 1e-12 if precision == "fp64" else 1e-5
    s, fresh = (gpu.CppStructuredSweepSession(g.wire(), g.structured(), g.X_flat(), dim=d, precision=precision)
                for _ in range(2))

    def same_report(E, M):
        fresh.set_X(s.get_X())
        assert (E[-1], M[-1]) == fresh.energy()

    E, M = s.run(1, omega=0.9)
    assert np.abs(s.get_X().reshape(-1, d) - Xo).max() <= tol
    same_report(E, M)
    for k in (2, 3):  # reports of captured chunks, and the two buffers in turn
        same_report(*s.run(6, omega=0.9, report_every=k))
