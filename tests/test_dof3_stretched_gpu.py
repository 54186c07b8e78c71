"""3D sweeps on boxes of very unequal spacing, in every axis order, against the
NumPy-patch oracle, at the bounds that boxes of equal spacing hold."""

from __future__ import annotations

import dataclasses
import itertools

import numpy as np
import pytest

from oracle import oracle
from tests.test_dof3_gpu import _box, _turned_cubes

pytestmark = pytest.mark.gpu

SPACINGS = [(1.0, 0.1, 0.1), (1.0, 0.1, 0.01), (1.0, 0.03, 0.03), (1.0, 0.01, 0.01)]
PHASES = [("barrier", 0.0), ("shape_size", 0.0), ("untangle", 0.1)]


def _stretch(make, L):
    """The grid of unit cells scaled to spacing L and cells of volume 1, its
    noise to fractions of the shortest spacing."""
    flat = make(0.0)
    noise = make(0.15).X - flat.X
    L = np.asarray(L) / np.prod(L) ** (1 / 3)
    return dataclasses.replace(flat, X=flat.X * L + noise * L.min()), L.min()


def _check(gpu, g, h, phase, delta, omega, variants):
    """One sweep: fp64 sums in another order stay within 1e-12 of the shortest
    spacing, a mixed sweep within the 1e-5 of it that the mixed path promises."""
    Xo, Eo, _ = oracle.run3(g.X, oracle.patches_for(g.blocks, g.free, d=3), oracle.stencil_for(g.blocks, d=3), 1,
                            phase=phase, delta=delta, omega=omega)
    for precision, tol in (("fp64", 1e-12), ("mixed", 1e-5)):
        for variant in variants:
            s = gpu.CppStructuredSweepSession(g.wire(), g.structured(), g.X_flat(), dim=3, precision=precision)
            s.set_variant(variant)
            E, _ = s.run(1, phase=phase, delta=delta, omega=omega)
            assert np.abs(s.get_X().reshape(-1, 3) - Xo).max() <= tol * h, (precision, variant)
            np.testing.assert_allclose(E, Eo, rtol=1e-12 if precision == "fp64" else 1e-5)


@pytest.mark.parametrize("phase,delta", PHASES)
@pytest.mark.parametrize("L", SPACINGS, ids=str)
def test_stretched_boxes_match_oracle(gpu, L, phase, delta):
    for order in sorted(set(itertools.permutations(L))):
        g, h = _stretch(lambda frac: _box((6, 5, 7), frac), order)
        _check(gpu, g, h, phase, delta, 0.9, (0, 1))


@pytest.mark.parametrize("L", SPACINGS, ids=str)
def test_stretched_lattice_dofs_match_oracle(gpu, L):
    """The nodes of a face between two blocks, one of them turned."""
    for order in sorted(set(itertools.permutations(L))):
        g, h = _stretch(lambda frac: _turned_cubes((1, 2, 0), (0, 1, 1), frac), order)
        _check(gpu, g, h, "barrier", 0.0, 0.8, (0,))
