"""Tile passes of the exact mode (quantr_gb300/csrc/exact.cu): amplitudes equal the oracle's value
for value, with no tolerance, at the edges of the tiles and for every gate kind; programs with
Custom gates and registers that are not finite take the one-launch-per-gate path."""
import numpy as np
import pytest

from quantr_gb300 import _native as nat
from quantr_gb300 import workloads as W
from quantr_gb300.program import ProgramBuilder
from test_wide_host import _everything

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _lib(gpu_lib):
    yield


def _run(prog, reg=None):
    h = nat.Handle(prog.n, nat.QGPU_C128, nat.QGPU_MODE_EXACT)
    if reg is not None:
        h.upload(reg)
    before = h.launch_count()
    h.apply(prog.ops, prog.mats, prog.none)
    launches = h.launch_count() - before
    out = h.download()
    h.close()
    return out, launches


def _standard(n, seed):
    prog = _everything(n, seed)
    prog.ops = prog.ops[prog.ops["kind"] != nat.KIND["Custom"]]
    return prog


@pytest.mark.parametrize("n", [3, 5, 6, 7, 8, 12, 13, 14, 17])
def test_every_gate_kind(oracle, n):
    prog = _standard(n, n)
    r = np.random.default_rng(n)
    reg = r.standard_normal(1 << n) + 1j * r.standard_normal(1 << n)
    for register in (None, reg / np.linalg.norm(reg)):
        out, launches = _run(prog, register)
        ref = oracle.simulate(prog, engine=oracle.DENSE_PAR) if register is None else \
            oracle.simulate(prog, register, engine=oracle.DENSE_PAR)
        assert np.array_equal(out, ref)
        assert launches < len(prog.ops)


@pytest.mark.parametrize("n,layers", [(1, 3), (2, 3), (10, 6), (15, 4), (18, 2)])
def test_families(oracle, n, layers):
    if n < 3:
        b = ProgramBuilder(n)
        for w in range(n):
            for g in ("Ry", "Rz", "Rx", "H"):
                b.add(g, w, (), param=0.4 + w if g[0] == "R" else 0.0)
        prog = b.build()
    else:
        prog = W.brickwork_qft(n=n, layers=layers, seed=7)
    out, _ = _run(prog)
    assert np.array_equal(out, oracle.simulate(prog, engine=oracle.DENSE_PAR))


def test_custom_gates_between(oracle):
    prog = _everything(9, 77)
    out, _ = _run(prog)
    assert np.array_equal(out, oracle.simulate(prog, engine=oracle.DENSE_PAR))


def test_many_gates_on_few_wires(oracle):
    """More gates than one pass's table holds."""
    b = ProgramBuilder(4)
    r = np.random.default_rng(2)
    for i in range(500):
        b.add(["Rx", "Ry", "Rz", "T"][i % 4], i % 4, (), param=r.uniform(-3, 3))
    prog = b.build()
    out, launches = _run(prog)
    assert np.array_equal(out, oracle.simulate(prog, engine=oracle.DENSE))
    assert launches >= 3


def test_registers_that_are_not_finite(oracle):
    """Products with 0 matter next to an infinity: the reference's NaNs appear."""
    n = 8
    reg = np.zeros(1 << n, np.complex128)
    reg[3] = 1.0
    reg[5] = np.inf
    b = ProgramBuilder(n)
    b.add("H", 2)
    b.add("CNot", 1, (7,))
    b.add("T", 5)
    prog = b.build()
    out, launches = _run(prog, reg)
    assert launches >= len(prog.ops)
    assert np.array_equal(out, oracle.simulate(prog, reg, engine=oracle.DENSE), equal_nan=True)


@pytest.mark.parametrize("angle", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("kind", ["CR", "Rz", "Ry"])
def test_angles_that_are_not_finite(oracle, kind, angle):
    """A NaN that a gate's entry brings in spreads through the products with 0 of the gates after it
    (H, H, CR(NaN), CNot: all four amplitudes)."""
    b = ProgramBuilder(3)
    for w in range(3):
        b.add("H", w)
    if kind == "CR":
        b.add("CR", 1, (0,), param=angle)
    else:
        b.add(kind, 1, (), param=angle)
    b.add("CNot", 2, (1,))
    b.add("T", 0)
    prog = b.build()
    out, _ = _run(prog)
    ref = oracle.simulate(prog, engine=oracle.DENSE)
    assert np.isnan(ref).any()
    assert np.array_equal(out, ref, equal_nan=True)
