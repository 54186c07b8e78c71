"""The grouped 3D forms of the sweep kernels (egg_b200/csrc/dof3.cuh), compiled
for the host, against extended precision: Newton step, gradient, metric change
and energy of a trial on boxes of equal and of very unequal spacing, in every
axis order, and on sheared cells."""

from __future__ import annotations

import shutil
import subprocess

import pytest

from tests.conftest import ROOT

# index of the cells in the program's output: spacings (3 axis orders each), then shear
CELLS = {0: "1:1:1", 15: "sheared"}
CELLS.update({3 * c + t: f"{s} order {t}"
              for c, s in ((1, "1:0.1:0.1"), (2, "1:0.1:0.01"), (3, "1:0.03:0.03"), (4, "1:0.01:0.01"))
              for t in range(3)})


@pytest.fixture(scope="module")
def report(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    exe = tmp_path_factory.mktemp("dof3") / "check"
    subprocess.run([gxx, "-O1", "-std=c++17", "-ffp-contract=off", f"-I{ROOT / 'egg_b200' / 'csrc'}",
                    str(ROOT / "tests" / "native" / "dof3_check.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    rows, same = {}, {}
    for line in out.strip().split("\n"):
        name, *f = line.split()
        if name == "same":
            same[f[0]] = float(f[1])
        else:
            rows[(name, int(f[0]), int(f[1]))] = tuple(float(v) for v in f[2:])
    return rows, same


@pytest.mark.parametrize("cells", sorted(CELLS), ids=lambda c: CELLS[c])
def test_grouped_forms_keep_the_plain_forms_accuracy(report, cells):
    """Where a cell's edges differ in length, products of lengths are larger
    than what the metric needs by (long / short)^2, so a form that subtracts
    them shows here as a hundred to a million times the plain form's error.
    Forms of cross products and sums of squares round like the plain ones:
    the factor 2 leaves room for the other order of the sums."""
    rows, _ = report
    for (name, at, kind), (median, p99, plain_median, plain_p99) in rows.items():
        if at != cells or name == "trial64":
            continue
        assert median <= 2 * plain_median, (name, kind)
        assert p99 <= 2 * plain_p99, (name, kind)
        if name.startswith("step") and cells != 15:  # the sweeps' own bounds, of the shortest spacing
            assert p99 <= (1e-5 if name == "step32" else 1e-12), (name, kind)


def test_trial_energies_round_like_their_sum(report):
    """Some 60 roundings of terms of one sign: 8 eps of the energy and its 32 ones."""
    rows, _ = report
    worst = [v[1] for (name, _, _), v in rows.items() if name == "trial64"]
    assert len(worst) == 3 * 13 + 2
    assert max(worst) <= 8 * 2.0**-52


def test_gradient_passes_skip_the_hessian_only(report):
    """The gradient-only pass (FAS restriction) forms the same sums."""
    _, same = report
    assert same == {"grad32": 0.0, "grad64": 0.0}
