"""One Newton step of the control-net PCG at the sizes its cluster of CTAs
splits unevenly (4 free controls; 4216, more than one per thread), against the
same step by torch autograd and a plain CG; and a batch's set_X from a mix of
page-locked and ordinary arrays."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from egg_b200 import configs, control

pytestmark = pytest.mark.gpu


def _energy(X):
    """Sum of mu - the 2D shape metric - over every corner sample of a block."""
    e = 0.0
    n = X.shape[0], X.shape[1]
    for b in range(4):
        i, j = b >> 1, b & 1

        def at(u, v):
            return X[u:n[0] - 1 + u, v:n[1] - 1 + v]

        c = at(i, j)
        e0 = (at(1 - i, j) - c) * (-1.0 if i else 1.0)
        e1 = (at(i, 1 - j) - c) * (-1.0 if j else 1.0)
        det = e0[..., 0] * e1[..., 1] - e1[..., 0] * e0[..., 1]
        e = e + ((e0 ** 2).sum(-1) + (e1 ** 2).sum(-1)).div(2 * det).sub(1).sum()
    return e


@pytest.mark.parametrize("net", [(4, 4), (66, 68)], ids=str)
def test_newton_step_matches_autograd(gpu, net):
    g = configs.unit_square(97, frac=0.1, seed=5)
    X0 = control.grid_block_nodes(g, 0)
    w = control.control_wire(X0, net)
    bases = [torch.from_numpy(np.ascontiguousarray(B)) for B in control.axis_bases(X0.shape[:-1], net)]
    b = torch.from_numpy(w["b"].reshape(X0.shape))
    C0 = torch.from_numpy(w["C0"].reshape(*net, 2))
    free = torch.zeros(net, dtype=torch.bool)
    free.reshape(-1)[torch.from_numpy(w["free_idx"].astype(np.int64))] = True

    def f(d):
        C = C0.clone()
        C[free] = C0[free] + d
        return _energy(torch.einsum("ia,jb,abc->ijc", bases[0], bases[1], C) + b)

    z = torch.zeros((int(free.sum()), 2), dtype=torch.float64)
    G = torch.autograd.functional.jacobian(f, z)

    def hv(v):
        return torch.autograd.functional.vhp(f, z, v)[1]

    x, r = torch.zeros_like(z), -G
    p, rr = r.clone(), float((r * r).sum())
    stop = 1e-26 * rr
    for _ in range(4000):
        q = hv(p)
        a = rr / float((p * q).sum())
        x, r = x + a * p, r - a * q
        new = float((r * r).sum())
        if new <= stop:
            break
        p, rr = r + (new / rr) * p, new
    s = gpu.CppStructuredSweepSession(g.wire(), g.structured(), g.X_flat(), control=w)
    rep = s.run_control(1, pcg_max_iter=4000, pcg_rtol=1e-13, pcg_forcing=False)
    assert rep["alphas"][0] == 1.0
    got = torch.from_numpy(s.get_C().reshape(*net, 2))[free] - C0[free]
    # both solve A dC = -G to 1e-13 of |G|; the energy's condition number on
    # these nets is below 1e5
    assert float((got - x).abs().max()) <= 1e-7 * float(x.abs().max())


def test_batch_set_x_takes_any_mix_of_arrays(gpu):
    ms = configs.batch_meshes(5, seed=3, hi=33)
    s = gpu.CppBatchSweepSession([(g.wire(compact=True), g.structured(), g.X_flat()) for g in ms])
    rng = np.random.default_rng(0)
    new = [g.X_flat() + 1e-3 * rng.normal(size=g.X.size) for g in ms]
    mixed = []
    for k, x in enumerate(new):
        if k % 2:
            t = torch.empty(x.size, dtype=torch.float64, pin_memory=True)
            t.copy_(torch.from_numpy(x))
            mixed.append(t.numpy())
        else:
            mixed.append(x)
    for arrays in (new, mixed, [list(x) for x in new]):
        s.set_X([np.zeros(x.size) for x in new])
        s.set_X(arrays)
        got = s.get_X()
        assert all(np.array_equal(a, x) for a, x in zip(got, new))
    got[0][:] = 7.0  # the views are the caller's own
    assert all(np.array_equal(a, x) for a, x in zip(s.get_X(), new))
    with pytest.raises(ValueError, match="one array per mesh"):
        s.set_X(new[:-1])
    with pytest.raises(ValueError, match="wrong length"):
        s.set_X([x[:-1] for x in new])
