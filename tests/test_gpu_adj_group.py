"""Grouped passes of the adjoint sweep (quantr_gb300/csrc/adj_group.cu) against the one-gate f64
sweep (QGPU_MODE_F64), at the edges of their tiles, for runs whose undo needs every part of the
frame: Y sums alone, X sums, both diagonals, a diagonal or antidiagonal undo, the -I sum.

Tolerances: complex128 1e-11 (float pairs, the adjoint tests' bar between sweep forms is 1e-9);
complex64 1e-4, the adjoint tests' bar.
"""
import numpy as np
import pytest

from quantr_gb300 import _native as nat
from quantr_gb300 import gradients as GR
from quantr_gb300.program import ProgramBuilder

pytestmark = pytest.mark.gpu

RUNS = {
    "ry_rz": ["Ry", "Rz"],
    "rz_ry": ["Rz", "Ry"],
    "rx": ["Rx"],
    "zyz": ["Rz", "Ry", "Rz"],
    "diagonal": ["Rz", "S", "T"],
    "antidiagonal": ["X", "Rz", "Y"],
    "phase": ["Phase", "Rx", "H"],
    "mixed": ["H", "Ry", "T", "Rx", "Phase", "X90"],
}


@pytest.fixture(autouse=True)
def _lib(gpu_lib):
    yield


def _program(n, run, seed):
    r = np.random.default_rng(seed)
    b = ProgramBuilder(n)
    for _ in range(2):
        for w in range(n):
            if run == "some" and w % 3 == 1:
                continue
            for g in RUNS[list(RUNS)[w % len(RUNS)] if run == "some" else run]:
                b.add(g, w, (), param=r.uniform(-3, 3) if g in ("Rx", "Ry", "Rz", "Phase") else 0.0)
        for w in range(n - 1):
            b.add("CNot", w + 1, (w,))
    return b.build(), r.standard_normal(n), r.standard_normal(n)


# 1, 2: below a round's bits; 8/9: thread bits / register bits; 11/12: one tile / two passes;
# 14: a last round of one wire
@pytest.mark.parametrize("n,run", [(1, "mixed"), (2, "zyz"), (3, "rx"), (5, "phase"), (8, "ry_rz"),
                                   (9, "mixed"), (11, "zyz"), (12, "rz_ry"), (13, "diagonal"),
                                   (13, "antidiagonal"), (14, "some"), (17, "mixed"), (21, "ry_rz")])
@pytest.mark.parametrize("precision", [nat.QGPU_C128, nat.QGPU_C64])
def test_grouped_passes_against_the_f64_sweep(monkeypatch, n, run, precision):
    monkeypatch.setenv("QGPU_ADJ_GROUP", "1")
    prog, a, b = _program(n, run, n)
    e, g = GR.energy_and_gradient(nat.Handle(n, precision), prog, a, b)
    re, rg = GR.energy_and_gradient(nat.Handle(n, nat.QGPU_C128, nat.QGPU_MODE_F64), prog, a, b)
    tol = 1e-11 if precision == nat.QGPU_C128 else 1e-4
    assert abs(e - re) <= tol
    assert np.max(np.abs(g - rg)) <= tol


@pytest.mark.parametrize("n", [21, 27])
def test_z_sums_of_registers_with_few_values(n):
    """Phases on low wires alone and no ZZ terms: a thread's products over its tiles are equal, and so
    are their rounding errors. The Z sums (Rz) and the -I sum (Phase) against the f64 sweep. Bar, in
    units of S = sum|x|: 2^-47 for a product of two float pairs, and the rounding of both vectors,
    2^-49 for each of the n + 5 gates each way, which equal amplitudes share: 1.2e-13 for n = 27, of which
    1e-13 is allowed."""
    b = ProgramBuilder(n)
    for w in range(n):
        b.add("H", w)
    b.add("Ry", n - 1, (), param=0.3)
    b.add("Rz", n - 1, (), param=0.7)
    b.add("Phase", n - 1, (), param=0.4)
    b.add("Rz", n - 2, (), param=0.2)
    b.add("Rz", n - 5, (), param=-0.5)
    prog = b.build()
    x = np.random.default_rng(n).uniform(0.5, 1.0, n)
    e, g = GR.energy_and_gradient(nat.Handle(n), prog, np.zeros(n), x)
    re, rg = GR.energy_and_gradient(nat.Handle(n, nat.QGPU_C128, nat.QGPU_MODE_F64), prog, np.zeros(n), x)
    assert abs(e - re) <= 1e-13 * x.sum()
    assert np.max(np.abs(g - rg)) <= 1e-13 * x.sum()
