"""A report launches no more CTAs than its cells fill; the allocation-free
energy always launches as many as fit.  The empty partials add nothing, so the
two agree bit for bit at every size."""

from __future__ import annotations

import pytest

from egg_b200 import configs

pytestmark = pytest.mark.gpu


# 225, 256 and 289 cells (256 a CTA); 151321 and 152100 (592 CTAs hold 151552)
@pytest.mark.parametrize("n", [2, 16, 17, 18, 390, 391])
def test_energy_equals_full_grid_2d(gpu, n):
    g = configs.unit_square(n, frac=0.25, seed=n)
    s = gpu.CppStructuredSweepSession(g.wire(compact=True), g.structured(), g.X_flat())
    assert s.energy() == s.energy_noalloc()
    if n > 2:
        E, M = s.run(2, report_every=2)
        assert (E[-1], M[-1]) == s.energy_noalloc()


# 64, 512 and 216 cells; 148877 and 157464
@pytest.mark.parametrize("n", [5, 9, 7, 54, 55])
def test_energy_equals_full_grid_3d(gpu, n):
    g = configs.unit_cube(n, frac=0.15, seed=n)
    s = gpu.CppStructuredSweepSession(g.wire(compact=True), g.structured(), g.X_flat(), dim=3)
    assert s.energy() == s.energy_noalloc()
    E, M = s.run(2, report_every=2)
    assert (E[-1], M[-1]) == s.energy_noalloc()
