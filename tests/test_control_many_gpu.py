"""Control nets of a batch against the same nets solved one by one: more
controls than the pull-back has warps, so that a warp takes several, and nets
that finish early beside nets that go on."""

from __future__ import annotations

import numpy as np
import pytest

from egg_b200 import configs, control

pytestmark = pytest.mark.gpu


def _warped(g, k):
    """Mesh k: the square bent by an amount that grows with k, so that the nets
    need different numbers of iterations."""
    x, y = g.X[:, 0], g.X[:, 1]
    bump = 0.02 * (k % 5) * np.sin(np.pi * x) * np.sin(np.pi * y)
    return np.ascontiguousarray(np.stack([x + bump, y - 0.5 * bump], axis=1))


@pytest.mark.parametrize("count", [2, 13, 400])  # one control a warp, up to two, more than 32
def test_batch_of_nets_equals_single_nets(gpu, count):
    g = configs.unit_square(65, frac=0.0)
    net = (59, 59)  # 57^2 free controls: 148 * 64 * 4 warps take 11 such nets at one control each
    wire, tables = g.wire(compact=True), g.structured()
    kinds = [_warped(g, k) for k in range(5)]
    cw = [control.control_wire(X.reshape(65, 65, 2), net) for X in kinds]
    b = gpu.CppBatchSweepSession([(wire, tables, kinds[m % 5].ravel()) for m in range(count)],
                                 control=[cw[m % 5] for m in range(count)])
    reps = b.run_control(2)
    X = b.get_X()
    for k in range(min(5, count)):
        s = gpu.CppStructuredSweepSession(wire, tables, kinds[k].ravel(), control=cw[k])
        one = s.run_control(2)
        for m in range(k, count, 5):
            assert list(reps[m]["pcg_iters"]) == list(one["pcg_iters"])
            np.testing.assert_array_equal(X[m], s.get_X())
