"""What a user of this framework has it do, as cases that can be timed.

Every case goes through the public entry points: a session built once from a
grid's wire, then per pass the upload of new positions from page-locked host
memory, the sweeps (or V-cycles, or control-net iterations) with their energy
reports, and the download of the positions.

fp64 sessions return positions and reports as they are (fp64).  Mixed sessions
compute their steps in fp32, and a program that asks for them holds its mesh in
fp32, so their results are returned in fp32.
"""

from __future__ import annotations

import functools
import math

import numpy as np
import torch

from egg_b200 import configs, control, cpp_core

DEVICE = "cuda:0"


def listed():
    return [
        # an interactive edit of a small O-grid: a few sweeps, then look at it again
        {"name": "disk17_edit", "kind": "sweep", "grid": "disk", "n": 17, "precision": "fp64", "phase": "barrier",
         "sweeps": 5, "report": 5, "frac": 0.25},
        # the 5-block O-H disk smoothed by 40 sweeps, two reports
        {"name": "disk65_smooth", "kind": "sweep", "grid": "disk", "n": 65, "precision": "fp64", "phase": "barrier",
         "sweeps": 40, "report": 20, "frac": 0.25},
        # boundary nodes sliding on their circle arcs while the disk is smoothed
        {"name": "disk129_slide", "kind": "slide", "n": 129, "precision": "fp64", "sweeps": 40, "report": 20},
        # the default precision on an ordinary single block, reports for a convergence plot
        {"name": "square1025_fp64", "kind": "sweep", "grid": "square", "n": 1025, "precision": "fp64",
         "phase": "barrier", "sweeps": 50, "report": 10, "frac": 0.3},
        # the largest 2D block, mixed precision
        {"name": "square4097_mixed", "kind": "sweep", "grid": "square", "n": 4097, "precision": "mixed",
         "phase": "barrier", "sweeps": 60, "report": 20, "frac": 0.3},
        # repair of a tangled block: one delta step of the untangle, then shape+size sweeps
        {"name": "square1025_repair", "kind": "repair", "n": 1025, "precision": "mixed", "sweeps": 40},
        # FAS V(2,2) cycles on a 2D block, default precision
        {"name": "square513_fas", "kind": "fas", "grid": "square", "n": 513, "precision": "fp64", "cycles": 4,
         "levels": 32, "frac": 0.25},
        # 256-mesh batches are swept in slices like this one: many meshes of uneven blocks, one session
        {"name": "batch48_mixed", "kind": "batch", "meshes": 48, "precision": "mixed", "sweeps": 20},
        # a 64 x 64 control net on one block: reduced Gauss-Newton
        {"name": "control64", "kind": "control", "n": 257, "net": 64, "precision": "fp64", "outer": 5},
        # 3D hex blocks around a sphere, default precision
        {"name": "sphere33_fp64", "kind": "sweep", "grid": "sphere", "n": 33, "precision": "fp64", "phase": "barrier",
         "sweeps": 10, "report": 10, "frac": 0.08},
        # one large hex block, mixed precision
        {"name": "cube129_mixed", "kind": "sweep", "grid": "cube", "n": 129, "precision": "mixed", "phase": "barrier",
         "sweeps": 20, "report": 10, "frac": 0.2},
        # FAS on the 7-block sphere-in-cube, mixed precision
        {"name": "sphere65_fas", "kind": "fas", "grid": "sphere", "n": 65, "precision": "mixed", "cycles": 2,
         "levels": 4, "frac": 0.08},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "slide", "repair", "fas", "batch", "control"])
    precision = rng.choice(["fp64", "mixed"])
    if kind == "sweep":
        grid = rng.choice(["disk", "square", "square", "sphere", "cube"])
        lo, hi = {"disk": (9, 400), "square": (17, 3000), "sphere": (7, 45), "cube": (9, 129)}[grid]
        n = _log_int(rng, lo, hi)
        sweeps = rng.randint(3, 60)
        report = rng.choice([sweeps, max(1, sweeps // 3)])
        return {"kind": kind, "grid": grid, "n": n, "precision": precision, "phase": "barrier", "sweeps": sweeps,
                "report": report, "frac": 0.08 if grid == "sphere" else rng.choice([0.15, 0.2, 0.25])}
    if kind == "slide":
        sweeps = rng.randint(5, 60)
        return {"kind": kind, "n": _log_int(rng, 9, 200), "precision": precision, "sweeps": sweeps, "report": sweeps}
    if kind == "repair":
        return {"kind": kind, "n": _log_int(rng, 33, 1400), "precision": precision, "sweeps": rng.randint(10, 60)}
    if kind == "fas":
        grid = rng.choice(["square", "sphere"])
        n = 8 * _log_int(rng, 4, 120) + 1 if grid == "square" else 4 * _log_int(rng, 2, 12) + 1
        return {"kind": kind, "grid": grid, "n": n, "precision": precision, "cycles": rng.randint(1, 4),
                "levels": rng.choice([3, 4, 32]), "frac": 0.08 if grid == "sphere" else 0.25}
    if kind == "batch":
        return {"kind": kind, "meshes": _log_int(rng, 2, 48), "precision": precision, "sweeps": rng.randint(5, 40)}
    return {"kind": kind, "n": _log_int(rng, 33, 300), "net": rng.randint(8, 30), "precision": precision,
            "outer": rng.randint(2, 5)}


# --- grids ------------------------------------------------------------------


def _spacing(blocks, X):
    """Shortest incident grid edge of every node."""
    h = np.full(X.shape[0], np.inf)
    for ids in blocks:
        for ax in range(ids.ndim):
            a = np.moveaxis(ids, ax, 0)[:-1].reshape(-1)
            b = np.moveaxis(ids, ax, 0)[1:].reshape(-1)
            ln = np.sqrt(((X[a] - X[b]) ** 2).sum(axis=1))
            o = np.argsort(ln)[::-1]  # the shortest is written last
            for v in (a, b):
                m = np.full_like(h, np.inf)
                m[v[o]] = ln[o]
                np.minimum(h, m, out=h)
    return h


class _Topology:
    """A grid without noise, its wire and block tables: the same for every seed."""

    def __init__(self, g, *, spacing=None, device=DEVICE):
        self.d, self.blocks, self.X, self.free = g.d, g.blocks, g.X, g.free
        self.h = spacing if spacing is not None else _spacing(g.blocks, g.X)
        self.wire = g.wire(compact=True, device=device)
        self.tables = g.structured()

    def noisy(self, frac, seed):
        """Positions with uniform noise of +-frac of the local spacing on the moving nodes."""
        X = torch.from_numpy(np.ascontiguousarray(self.X)).to(DEVICE)
        rng = torch.Generator(device=DEVICE).manual_seed(seed)
        u = torch.rand(X.shape, generator=rng, dtype=torch.float64, device=DEVICE) * 2 - 1
        h = torch.as_tensor(self.h, dtype=torch.float64, device=DEVICE)
        amp = torch.from_numpy(self.free).to(DEVICE) * frac * h
        return (X + u * amp[:, None]).reshape(-1)


@functools.lru_cache(maxsize=6)
def _topology(grid, n):
    make = {"disk": configs.disk_oh, "square": configs.unit_square, "sphere": configs.sphere_in_cube,
            "cube": configs.unit_cube}[grid]
    g = make(n, frac=0.0)
    return _Topology(g, spacing=1.0 / (n - 1) if grid in ("square", "cube") else None)


@functools.lru_cache(maxsize=2)
def _batch_topology(count):
    return [_Topology(configs.multiblock_mesh(k, frac=0.0), spacing=1.0 / 256) for k in range(count)]


def _pinned(x):
    t = torch.empty(x.shape, dtype=torch.float64, pin_memory=True)
    t.copy_(x)
    return t


def _tangled(t, seed):
    """Noise-free positions with a few nodes thrown 0.8-1.5 spacings away, which inverts about 5% of the cells."""
    X = torch.from_numpy(np.ascontiguousarray(t.X)).to(DEVICE)
    rng = torch.Generator(device=DEVICE).manual_seed(seed)
    u = torch.rand((3, X.shape[0]), generator=rng, dtype=torch.float64, device=DEVICE)
    hit = torch.from_numpy(t.free).to(DEVICE) & (u[0] < 0.018)
    r, th = (0.8 + 0.7 * u[1]) * t.h, 2 * math.pi * u[2]
    step = torch.stack([r * torch.cos(th), r * torch.sin(th)], dim=1)
    return (X + step * hit[:, None]).reshape(-1)


def _mean_size_target(t):
    return configs.mean_size_w_inv(t.blocks, t.X)


def _repair_delta(t, X):
    """The first delta of the untangle schedule: twice the worst corner determinant."""
    cells = torch.from_numpy(_cells(t.blocks)).to(DEVICE)
    return 2.0 * abs(float(_energy(X.reshape(-1, 2), cells, "barrier", 0.0, None)[1]))


def _slide_grid(case, seed):
    return configs.disk_on_curve(case["n"], seed=seed, arcs=True)


def _warped(t, seed):
    """A smoothly distorted block with a little noise: what a net is fitted to."""
    rng = np.random.default_rng(seed)
    x, y = t.X[:, 0], t.X[:, 1]
    bump = np.sin(math.pi * x) * np.sin(math.pi * y)
    X = t.X.copy()
    for k in range(2):
        a, b, p = rng.uniform(0.5, 2.0), rng.uniform(0.5, 2.0), rng.uniform(0, 2 * math.pi)
        X[:, k] += 0.06 * bump * np.sin(2 * math.pi * (a * x + b * y) + p)
    return X + np.where(t.free[:, None], rng.uniform(-0.1, 0.1, X.shape) * t.h, 0.0)


def _session(t, X, precision, wire=None, **kw):
    return cpp_core.CppStructuredSweepSession(wire if wire is not None else t.wire, t.tables, X, device=DEVICE,
                                              dim=t.d, precision=precision, **kw)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        ts = _batch_topology(case["meshes"])
        Xs = [_pinned(t.noisy(0.25, seed * 1009 + k)) for k, t in enumerate(ts)]
        s = cpp_core.CppBatchSweepSession([(t.wire, t.tables, X.numpy()) for t, X in zip(ts, Xs)], device=DEVICE,
                                          dim=2, precision=case["precision"])
        return {"case": case, "s": s, "X": [X.numpy() for X in Xs], "keep": Xs}
    if kind == "slide":
        g = _slide_grid(case, seed)
        X = _pinned(torch.from_numpy(g.X_flat()))
        s = cpp_core.CppStructuredSweepSession(g.wire(compact=True), g.structured(), X.numpy(), device=DEVICE, dim=2,
                                               precision=case["precision"])
        return {"case": case, "s": s, "X": X.numpy(), "keep": X}
    if kind == "control":
        t = _topology("square", case["n"])
        X = _warped(t, seed)
        w = control.control_wire(X[t.blocks[0].reshape(-1)].reshape(t.blocks[0].shape + (2,)),
                                 (case["net"], case["net"]))
        s = _session(t, np.ascontiguousarray(X).reshape(-1), case["precision"], control=w)
        return {"case": case, "s": s, "C": w["C0"]}
    if kind == "repair":
        t = _topology("square", case["n"])
        x = _tangled(t, seed)
        X = _pinned(x)
        a = _session(t, X.numpy(), case["precision"])
        b = _session(t, X.numpy(), case["precision"], wire=_size_wire(case["n"]))
        return {"case": case, "s": a, "b": b, "X": X.numpy(), "keep": X, "delta": _repair_delta(t, x)}
    t = _topology(case["grid"], case["n"])
    X = _pinned(t.noisy(case["frac"], seed))
    return {"case": case, "s": _session(t, X.numpy(), case["precision"]), "X": X.numpy(), "keep": X}


@functools.lru_cache(maxsize=2)
def _size_wire(n):
    """The square's wire with the mean-size target of the shape+size phase."""
    t = _topology("square", n)
    return configs.unit_square(n, frac=0.0).wire(compact=True, w_inv=_mean_size_target(t), device=DEVICE)


def _result(case, **out):
    if case["precision"] == "fp64":
        return out
    return {k: [torch.from_numpy(x).float() for x in v] if isinstance(v, list) else torch.from_numpy(v).float()
            for k, v in out.items()}


def run(state):
    case, s = state["case"], state["s"]
    kind = case["kind"]
    if kind == "control":
        s.set_C(state["C"])
        r = s.run_control(case["outer"])
        return _result(case, X=s.get_X(), C=s.get_C(), E=np.asarray(r["energies"]))
    s.set_X(state["X"])
    if kind == "repair":
        E, M = s.run(20, phase="untangle", delta=state["delta"], omega=0.5)
        b = state["b"]
        b.set_X(s.get_X())
        E2, M2 = b.run(case["sweeps"], phase="shape_size")
        return _result(case, X=b.get_X(), E=np.concatenate([E, E2]), M=np.concatenate([M, M2]))
    if kind == "fas":
        E, M = s.run_fas(case["cycles"], nu_pre=2, nu_post=2, max_levels=case["levels"])
    elif kind == "batch":
        E, M = s.run(case["sweeps"], report_every=case["sweeps"])
        return _result(case, X=s.get_X(), E=np.asarray(E), M=np.asarray(M))
    else:
        E, M = s.run(case["sweeps"], phase=case.get("phase", "barrier"), report_every=case["report"])
    return _result(case, X=s.get_X(), E=E, M=M)


# --- what a pass cannot do without -------------------------------------------

# Floating-point operations of one vertex update.  2D: the four samples of one
# cell (each counted once) with the gradient and Hessian parts of their three
# nodes (about 110 each), the solve, and one trial over the 12 moving samples
# (about 25 each).  3D: eight samples of about 100 with four nodes of about 60
# each, the solve, and one trial over 32 moving samples (about 45 each).
FLOPS_UPDATE = {2: 780, 3: 4250}
# One sample's metric in an energy report.
FLOPS_SAMPLE = {2: 12, 3: 70}


def _count(case):
    """(nodes, moving nodes, cells, dimension)"""
    if case["kind"] == "batch":
        # the mean mesh: 6 blocks of about 90 x 90
        k = case["meshes"]
        return k * 47700, k * 46600, k * 47000, 2
    n, grid = case["n"], case.get("grid", "disk" if case["kind"] == "slide" else "square")
    return {"square": (n * n, (n - 2) ** 2, (n - 1) ** 2, 2),
            "disk": (5 * n * n, 5 * (n - 1) ** 2, 5 * (n - 1) ** 2, 2),
            "cube": (n**3, (n - 2) ** 3, (n - 1) ** 3, 3),
            "sphere": (7 * n**3, 7 * (n - 1) ** 3, 7 * (n - 1) ** 3, 3)}[grid]


def work(case):
    nodes, moving, cells, d = _count(case)
    sample = cells * 2**d * FLOPS_SAMPLE[d]
    bytes_ = 2 * nodes * d * 8
    kind = case["kind"]
    if kind == "control":
        # per outer iteration about 10 CG products, each one pass over the cells' samples; two energies
        flops = case["outer"] * (10 * 4 * sample + 2 * sample)
        bytes_ = nodes * d * 8 + 2 * case["net"] ** 2 * d * 8
    elif kind == "fas":
        # 4 fine sweeps and 2 gradient passes a cycle, the coarser levels' share, 3 energies
        level = 1 / (1 - 2.0**-d)
        flops = case["cycles"] * (moving * FLOPS_UPDATE[d] * (4 * level + 2) + 3 * sample)
    else:
        sweeps = case["sweeps"] + (20 if kind == "repair" else 0)
        reports = 2 if kind == "repair" else -(-case["sweeps"] // case.get("report", case["sweeps"]))
        flops = moving * FLOPS_UPDATE[d] * sweeps + reports * sample
    return {"bytes": float(bytes_), "flops": float(flops)}


# --- the same sweeps in 64 bits, by torch alone -------------------------------
#
# One sweep relaxes every moving node on the frozen positions: the Newton step
# of its patch energy (every corner sample of every cell around it), halved up
# to ten times until the patch energy does not grow and, outside the untangle
# phase, no corner determinant is negative.


def _cells(blocks):
    """Corner node ids of every cell, (cells, 2^d), corner bits with axis 0 first."""
    out = []
    for ids in blocks:
        d = ids.ndim
        c = [ids[tuple(slice(1, None) if (b >> (d - 1 - k)) & 1 else slice(0, -1) for k in range(d))].reshape(-1)
             for b in range(1 << d)]
        out.append(np.stack(c, axis=1))
    return np.concatenate(out).astype(np.int64)


def _columns(P, b, d):
    """(signed edges, signs) of corner sample b of cells with corner positions P[corner] (n, d)."""
    e, s = [], []
    for k in range(d):
        bit = 1 << (d - 1 - k)
        s.append(-1.0 if b & bit else 1.0)
        e.append((P[b ^ bit] - P[b]) * s[-1])
    return e, s


def _dot(a, b):
    return (a * b).sum(dim=1)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=1)


def _scale(D, phase, delta):
    """f, f', f'' of the determinant: 1/(2D), or its untangle surrogate, times 2 (so 1/Dh and its derivatives)."""
    if phase == "untangle":
        r = torch.sqrt(D * D + 4 * delta * delta)
        Dh, d1, d2 = 0.5 * (D + r), 0.5 * (1 + D / r), 2 * delta * delta / r**3
    else:
        Dh, d1, d2 = D, torch.ones_like(D), torch.zeros_like(D)
    return Dh, d1, d2


def _parts(e, d):
    s = sum(_dot(x, x) for x in e)
    if d == 2:
        C = [torch.stack([e[1][:, 1], -e[1][:, 0]], dim=1), torch.stack([-e[0][:, 1], e[0][:, 0]], dim=1)]
    else:
        C = [_cross(e[1], e[2]), _cross(e[2], e[0]), _cross(e[0], e[1])]
    D = _dot(e[0], C[0])
    q = sum(_dot(c, c) for c in C) if d == 3 else None
    return s, q, C, D


def _value(e, d, phase, delta):
    s, q, _, D = _parts(e, d)
    Dh = _scale(D, phase, delta)[0]
    m = s / (2 * Dh) if d == 2 else s * q / (9 * Dh * Dh)
    if phase == "shape_size":
        return (m * m if d == 2 else m) - 1 + (D - 1) ** 2, D
    return m - 1, D


def _node_parts(e, signs, role, d, phase, delta):
    """Gradient (n, d) and Hessian (n, d, d) of one sample for the node in `role` (0 corner, 1 + k its axis-k neighbour)."""
    v = [-x for x in signs] if role == 0 else [signs[k] if k == role - 1 else 0.0 for k in range(d)]
    s, q, C, D = _parts(e, d)
    a = sum(v[k] * e[k] for k in range(d) if v[k])
    c = sum(v[k] * C[k] for k in range(d) if v[k])
    vv = sum(x * x for x in v)
    Dh, d1, d2 = _scale(D, phase, delta)
    eye = torch.eye(d, dtype=e[0].dtype, device=e[0].device)

    def outer(x, y):
        return x[:, :, None] * y[:, None, :]

    def sym(x, y):
        o = outer(x, y)
        return o + o.transpose(1, 2)

    def w(x):
        return x[:, None, None]

    if d == 2:
        f, f1 = 0.5 / Dh, -0.5 * d1 / Dh**2
        f2 = -0.5 * d2 / Dh**2 + d1 * d1 / Dh**3
        g = 2 * f[:, None] * a + (s * f1)[:, None] * c
        H = w(2 * vv * f) * eye + w(2 * f1) * sym(a, c) + w(s * f2) * outer(c, c)
        if phase == "shape_size":
            m = s * f
            H = 2 * outer(g, g) + w(2 * m) * H + 2 * outer(c, c)
            g = 2 * m[:, None] * g + 2 * (D - 1)[:, None] * c
        return g, H
    F, F1 = 1 / Dh**2, -2 * d1 / Dh**3
    F2 = 6 * d1 * d1 / Dh**4 - 2 * d2 / Dh**3
    G = sum(outer(x, x) for x in e)
    k = s[:, None] * a - sum(_dot(x, a)[:, None] * x for x in e)
    m = w(vv * s - _dot(a, a)) * eye - vv * G + outer(a, a)
    g = (2 * (q * F)[:, None] * a + 2 * (s * F)[:, None] * k + (s * q * F1)[:, None] * c) / 9
    H = (w(2 * vv * q * F) * eye + w(2 * s * F) * m + w(s * q * F2) * outer(c, c) + w(4 * F) * sym(a, k)
         + w(2 * q * F1) * sym(a, c) + w(2 * s * F1) * sym(k, c)) / 9
    if phase == "shape_size":
        g, H = g + 2 * (D - 1)[:, None] * c, H + 2 * outer(c, c)
    return g, H


def _chunks(n, size=1 << 20):
    return [slice(i, min(n, i + size)) for i in range(0, n, size)]


def _energy(X, cells, phase, delta, w):
    """(sum of the metric, smallest determinant) over every corner sample; w: a scalar target, T = w A."""
    d, E, M = X.shape[1], 0.0, None
    for c in _chunks(cells.shape[0]):
        P = [X[cells[c, b]] for b in range(1 << d)]
        for b in range(1 << d):
            e, _ = _columns(P, b, d)
            _, D = _value(e, d, "barrier", 0.0)
            mu, _ = _value([x * w for x in e] if w is not None else e, d, phase, delta)
            E = E + mu.sum()
            M = D.min() if M is None else torch.minimum(M, D.min())
    return E, M


def _solve(H, g):
    d = g.shape[1]
    if d == 2:
        adj = torch.stack([torch.stack([H[:, 1, 1], -H[:, 0, 1]], 1), torch.stack([-H[:, 1, 0], H[:, 0, 0]], 1)], 1)
        det = H[:, 0, 0] * H[:, 1, 1] - H[:, 0, 1] * H[:, 1, 0]
    else:
        r = [H[:, i] for i in range(3)]
        adj = torch.stack([_cross(r[1], r[2]), _cross(r[2], r[0]), _cross(r[0], r[1])], dim=2)
        det = _dot(r[0], adj[:, :, 0])
    x = -(adj * g[:, None, :]).sum(dim=2) / det[:, None]
    gn = g.norm(dim=1)
    x = torch.where(torch.isfinite(x).all(dim=1)[:, None], x, -0.1 * g / gn[:, None])
    return torch.where((gn < 1e-15)[:, None], torch.zeros_like(x), x)


def _patch_energy(X, cells, corner, move, phase, delta, e_sum, d_min):
    """Adds the energies of `cells` with the node at `corner` displaced by `move` (None: not) to that node's sums."""
    d = X.shape[1]
    node = cells[:, corner]
    P = [X[cells[:, b]] for b in range(1 << d)]
    if move is not None:
        P[corner] = P[corner] + move[node]
    e, md = 0.0, None
    for b in range(1 << d):
        mu, D = _value(_columns(P, b, d)[0], d, phase, delta)
        e, md = e + mu, D if md is None else torch.minimum(md, D)
    e_sum.index_add_(0, node, e)
    d_min.scatter_reduce_(0, node, md, "amin")


def _sweep(X, cells, moving, phase, delta, omega):
    N, d = X.shape
    kw = {"dtype": X.dtype, "device": X.device}
    g, H = torch.zeros((N, d), **kw), torch.zeros((N, d * d), **kw)
    e0, md = torch.zeros(N, **kw), torch.full((N,), math.inf, **kw)
    for c in _chunks(cells.shape[0]):
        P = [X[cells[c, b]] for b in range(1 << d)]
        for b in range(1 << d):
            e, signs = _columns(P, b, d)
            for role in range(d + 1):
                node = cells[c, b if role == 0 else b ^ (1 << (d - role))]
                gi, Hi = _node_parts(e, signs, role, d, phase, delta)
                g.index_add_(0, node, gi)
                H.index_add_(0, node, Hi.reshape(-1, d * d))
            _patch_energy(X, cells[c], b, None, phase, delta, e0, md)
    step = _solve(H.reshape(N, d, d), g)
    done, alpha = ~moving, 1.0
    out = X.clone()
    for _ in range(10):
        trial = alpha * step
        e, md = torch.zeros(N, **kw), torch.full((N,), math.inf, **kw)
        for b in range(1 << d):
            part = cells[~done[cells[:, b]]]
            for c in _chunks(part.shape[0]):
                _patch_energy(X, part[c], b, trial, phase, delta, e, md)
        ok = ~done & torch.isfinite(e) & (e <= e0 + 1e-12)
        if phase != "untangle":
            ok &= md > 0
        out = torch.where(ok[:, None], X + omega * trial, out)
        done = done | ok
        alpha *= 0.5
        if bool(done.all()):
            break
    return out


def _run64(X, cells, moving, sweeps, report, phase="barrier", delta=0.0, omega=1.0, w=None, parts=None):
    E, M = [], []
    for k in range(sweeps):
        X = _sweep(X, cells, moving, phase, delta, omega)
        if (k + 1) % report == 0 or k + 1 == sweeps:
            r = [_energy(X, c, phase, delta, w) for c in (parts or [cells])]
            E.append([float(e) for e, _ in r])
            M.append([float(m) for _, m in r])
    E, M = np.array(E), np.array(M)
    return X, (E if parts else E[:, 0]), (M if parts else M[:, 0])


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("sweep", "repair", "batch"):
        return None  # V-cycles, nets and boundary curves: too long to restate here
    if kind == "batch":
        ts = _batch_topology(case["meshes"])
        X = torch.cat([t.noisy(0.25, seed * 1009 + k) for k, t in enumerate(ts)]).reshape(-1, 2)
        at, parts = 0, []
        for t in ts:
            parts.append(torch.from_numpy(_cells(t.blocks) + at).to(DEVICE))
            at += t.X.shape[0]
        moving = torch.from_numpy(np.concatenate([t.free for t in ts])).to(DEVICE)
        X, E, M = _run64(X, torch.cat(parts), moving, case["sweeps"], case["sweeps"], parts=parts)
        return {"X": [x.reshape(-1) for x in X.split([t.X.shape[0] for t in ts])], "E": E, "M": M}
    t = _topology("square" if kind == "repair" else case["grid"], case["n"])
    cells = torch.from_numpy(_cells(t.blocks)).to(DEVICE)
    moving = torch.from_numpy(t.free).to(DEVICE)
    if kind == "repair":
        x = _tangled(t, seed)
        X, E, M = _run64(x.reshape(-1, 2), cells, moving, 20, 20, "untangle", _repair_delta(t, x), 0.5)
        w = float(_mean_size_target(t)[0, 0])
        X, E2, M2 = _run64(X, cells, moving, case["sweeps"], case["sweeps"], "shape_size", w=w)
        return {"X": X.reshape(-1), "E": np.concatenate([E, E2]), "M": np.concatenate([M, M2])}
    if moving.sum() * case["sweeps"] > 1.1e9:
        return None  # over 20 seconds
    x = t.noisy(case["frac"], seed).reshape(-1, t.d)
    X, E, M = _run64(x, cells, moving, case["sweeps"], case["report"], case["phase"])
    return {"X": X.reshape(-1), "E": E, "M": M}
