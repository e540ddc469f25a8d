"""Custom gates on one wire that grow the register: the bound on its amplitudes, which the digit passes
and the exact mode's tile passes rely on and which sends fast-mode programs past the float range to
f64 arithmetic, follows them. Bars: the parity tests' 1e-12 of the largest amplitude; the exact mode
value for value."""
import numpy as np
import pytest

from quantr_gb300 import _native as nat
from quantr_gb300 import workloads as W
from quantr_gb300.program import ProgramBuilder

pytestmark = pytest.mark.gpu
NONE = np.zeros(2, np.uint8)


@pytest.fixture(autouse=True)
def _lib(gpu_lib):
    yield


def _near(out, ref):
    assert np.max(np.abs(out - ref)) <= 1e-12 * np.max(np.abs(ref))


@pytest.mark.parametrize("growth", [1.0, 3.0, 1e3, 1e9])
@pytest.mark.parametrize("matrix", [np.eye(2), np.array([[0.6, 0.8], [-0.8, 0.6]])])
def test_digit_passes_of_the_next_program(monkeypatch, oracle, growth, matrix):
    monkeypatch.setenv("QGPU_DIGITS_MIN_QUBITS", "11")
    n = 14
    b = ProgramBuilder(n)
    b.add("Ry", 3, (), param=0.7)
    b.add_custom(4, [], (growth * matrix).astype(np.complex128), NONE)
    first, second = b.build(), W.brickwork_qft(n=n, layers=8, seed=5, qft=False)
    h = nat.Handle(n)
    h.set_profiling(True)
    for prog in (first, second):
        h.apply(prog.ops, prog.mats, prog.none)
    assert "k_dg2" in h.profile()
    ref = oracle.simulate(first, engine=oracle.DENSE_PAR)
    _near(h.download(), oracle.simulate(second, ref, engine=oracle.DENSE_PAR))
    h.close()


@pytest.mark.parametrize("growth", [1e10, 1e19, 1e25, 1e100])
def test_growth_past_the_float_range(oracle, growth):
    n = 12
    b = ProgramBuilder(n)
    for w in range(n):
        b.add("Ry", w, (), param=0.7)
    for w in (2, 5):  # (a phase on one wire, a map under a control)
        b.add_custom(w, [], np.diag([growth, growth * 1j]), NONE)
        m = np.eye(4, dtype=np.complex128)
        m[3, 3] = 0.5
        b.add_custom(w, [w + 1], m, np.zeros(4, np.uint8))
        b.add("CNot", (w + 1) % n, (w,))
    for w in range(n):
        b.add("Rx", w, (), param=0.7)
    prog = b.build()
    h = nat.Handle(n)
    h.apply(prog.ops, prog.mats, prog.none)
    _near(h.download(), oracle.simulate(prog, engine=oracle.DENSE_PAR))
    h.close()


def test_exact_mode_after_growth_to_infinity(oracle):
    n = 8
    b = ProgramBuilder(n)
    b.add("H", 2)
    b.add_custom(4, [], np.eye(2, dtype=np.complex128) * 1e200, NONE)
    grow = b.build()
    b = ProgramBuilder(n)
    for name, t, c in (("H", 2, ()), ("CNot", 1, (7,)), ("T", 5, ())):
        b.add(name, t, c)
    prog = b.build()
    h = nat.Handle(n, nat.QGPU_C128, nat.QGPU_MODE_F64)
    for _ in range(2):
        h.apply(grow.ops, grow.mats, grow.none)
    reg = h.download()
    assert np.isinf(reg.real).any()
    h.set_mode(nat.QGPU_MODE_EXACT)
    h.apply(prog.ops, prog.mats, prog.none)
    assert np.array_equal(h.download(), oracle.simulate(prog, reg, engine=oracle.DENSE), equal_nan=True)
    h.close()


@pytest.mark.parametrize("growth", [3.0, 1e6])
def test_growth_between_pair_passes(monkeypatch, oracle, growth):
    """Kept apart from the pair blocks by Toffoli gates: digits up to a growth of 16, float pairs past it."""
    monkeypatch.setenv("QGPU_DIGITS_MIN_QUBITS", "11")
    n = 14
    layers = W.brickwork_qft(n=n, layers=8, seed=6, qft=False)
    b = ProgramBuilder(n)
    for _ in range(2):
        b.add("Toffoli", 4, (1, 9))
        b.add_custom(4, [], np.eye(2, dtype=np.complex128) * growth ** 0.5, NONE)
    b.add("Toffoli", 4, (0, 7))
    grow = b.build()
    prog = _joined(layers, grow, layers)
    h = nat.Handle(n)
    h.set_profiling(True)
    h.apply(prog.ops, prog.mats, prog.none)
    assert ("k_dg2" in h.profile()) == (growth <= 16.0)
    _near(h.download(), oracle.simulate(prog, engine=oracle.DENSE_PAR))
    h.close()


def _joined(*programs):
    """One program of several, of which only one has Custom gates (their tables stay where they are)."""
    own = next(p for p in programs if p.mats.size)
    return type(own)(own.n, np.concatenate([p.ops for p in programs]), own.mats, own.none)
