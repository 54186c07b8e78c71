"""The three classes of the 3D stored-patch kernel: general patches alone,
lattice DOFs beside them, constrained DOFs beside both."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from egg_b200 import configs
from oracle import oracle

pytestmark = pytest.mark.gpu


def _halves(g):
    """The same mesh as two blocks that meet in the middle."""
    ids = g.blocks[0]
    m = ids.shape[0] // 2
    return dataclasses.replace(g, blocks=[ids[:m + 1], ids[m:]])


def _hmin(g):
    return float(configs._min_edge(g.blocks, g.X).min())


@pytest.mark.parametrize("target", ["general", "identity"])
@pytest.mark.parametrize("phase,delta", [("barrier", 0.0), ("shape_size", 0.0), ("untangle", 0.05)])
def test_free_classes_match_oracle(gpu, target, phase, delta):
    """A target that is no multiple of the identity stores every DOF's patch
    (class 0); the face between two blocks is a lattice (class 1).  fp64 sums in
    another order: 1e-12 of the spacing."""
    g = _halves(configs.unit_cube(7, frac=0.15, seed=2))
    g = dataclasses.replace(g, X=g.X * 6.0)  # unit spacing
    w = np.array([[1.0, 0.1, 0.0], [0.0, 1.1, 0.0], [0.05, 0.0, 0.9]]) if target == "general" else None
    Xo, Eo, _ = oracle.run3(g.X, oracle.patches_for(g.blocks, g.free, w_inv=w, d=3),
                            oracle.stencil_for(g.blocks, w_inv=w, d=3), 1, phase=phase, delta=delta, omega=0.9)
    s = gpu.CppStructuredSweepSession(g.wire(w_inv=w), g.structured(), g.X_flat(), dim=3)
    E, _ = s.run(1, phase=phase, delta=delta, omega=0.9)
    assert np.abs(s.get_X().reshape(-1, 3) - Xo).max() <= 1e-12
    np.testing.assert_allclose(E, Eo, rtol=1e-12)


@pytest.mark.parametrize("make", [configs.cube_sliding, configs.cube_curved], ids=lambda f: f.__name__)
def test_constrained_class_with_lattice_dofs(gpu, make):
    """A sliding cube cut in two relaxes as in one block: the nodes of the cut
    as lattice DOFs instead of tile DOFs, the sliding ones as before."""
    g = make(9)
    one, two = (gpu.CppStructuredSweepSession(x.wire(), x.structured(), x.X_flat(), dim=3) for x in (g, _halves(g)))
    for omega in (1.0, 0.8):  # the second call starts from the first one's feet
        one.run(1, omega=omega)
        two.run(1, omega=omega)
        assert np.abs(one.get_X() - two.get_X()).max() <= 1e-12 * _hmin(g)
