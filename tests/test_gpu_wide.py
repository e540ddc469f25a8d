"""Wide passes (quantr_gb300/csrc/wide.cuh) on the GPU against the oracle, at the edges of their
tiles: registers below a round's bits, below and at a tile, one bit past it; every gate kind, Custom
gates, controls and phase bits inside and outside the tile; an uploaded register.

Tolerances, the parity tests': complex128 1e-12 of the largest amplitude, complex64 1 - F <= 1e-8."""
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


def _check(oracle, prog, precision, reg=None):
    h = nat.Handle(prog.n, precision)
    h.set_profiling(True)
    if reg is not None:
        h.upload(reg)
    h.apply(prog.ops, prog.mats, prog.none)
    out = h.download()
    prof = h.profile()
    h.close()
    ref = oracle.simulate(prog, reg, engine=oracle.DENSE_PAR) if reg is not None else \
        oracle.simulate(prog, engine=oracle.DENSE_PAR)
    if precision == nat.QGPU_C128:
        assert np.max(np.abs(out - ref)) <= 1e-12 * max(1.0, np.max(np.abs(ref)))
    else:
        f = abs(np.vdot(ref, out)) ** 2 / (np.vdot(ref, ref).real * np.vdot(out, out).real)
        assert 1.0 - f <= 1e-8
    return prof


@pytest.mark.parametrize("precision", [nat.QGPU_C128, nat.QGPU_C64])
@pytest.mark.parametrize("n", [3, 4, 6, 9, 10, 11, 12, 14])
def test_every_gate_kind(oracle, n, precision):
    r = np.random.default_rng(n)
    reg = r.standard_normal(1 << n) + 1j * r.standard_normal(1 << n)
    prof = _check(oracle, _everything(n, n + 40), precision, reg / np.linalg.norm(reg))
    assert n < 9 or any(k.startswith("k_wide") for k in prof), prof  # (smaller: a tile pass holds it all)


@pytest.mark.parametrize("precision", [nat.QGPU_C128, nat.QGPU_C64])
@pytest.mark.parametrize("family,n", [("ansatz", 1), ("ansatz", 2), ("ansatz", 10), ("ansatz", 13),
                                      ("ansatz", 18), ("columns", 11), ("columns", 15), ("brickwork", 12),
                                      ("brickwork", 17), ("qft", 13), ("ansatz", 21)])
def test_families(oracle, family, n, precision):
    prog = {"ansatz": lambda: W.ansatz(n=n, layers=3, seed=1).program(),
            "columns": lambda: W.random_columns(n=n, columns=30, seed=2),
            "brickwork": lambda: W.brickwork_qft(n=n, layers=8, seed=3, qft=False),
            "qft": lambda: W.brickwork_qft(n=n, layers=2, seed=3)}[family]() if n > 2 else _small(n)
    prof = _check(oracle, prog, precision)
    assert n < 3 or any(k.startswith("k_wide") for k in prof), prof


def _small(n):
    from quantr_gb300.program import ProgramBuilder

    b = ProgramBuilder(n)
    for w in range(n):
        b.add("Ry", w, (), param=0.3 + w)
        b.add("Rz", w, (), param=-1.2)
    if n > 1:
        b.add("CNot", 1, (0,))
        b.add("Rx", 1, (), param=0.8)
        b.add("CNot", 0, (1,))
        b.add("Ry", 0, (), param=2.5)
    return b.build()


def _chain(kind, n, layers):
    """Custom gates that are nearly, but not exactly, unitary, in every layer."""
    r = np.random.default_rng(11)
    b = ProgramBuilder(n)
    none = np.zeros(2, np.uint8)
    c, s = np.cos(0.4), np.sin(0.4)
    matrix = {"real": np.full((2, 2), 0.7071067811865) * [[1, 1], [1, -1]],  # 13 digits of sqrt(1/2)
              "complex": (1.0 - 1.6e-13) * np.array([[c, -s], [1j * s, 1j * c]]),
              "phase": np.diag([1.0, 1.0 - 4e-13])}  # damps |1>
    matrix["grown"] = matrix["real"]
    for w in range(n):
        b.add("Ry", w, (), param=r.uniform(0.3, 2.8))
    for layer in range(layers):
        for w in range(n):
            b.add_custom(w, [], matrix[kind].astype(np.complex128), none)
            if kind == "grown" and layer == layers // 2:  # not unitary at all, in between
                b.add_custom(w, [], np.array([[1.25, 0.25], [-0.5, 0.75]], np.complex128), none)
            if kind == "phase":  # (Toffoli gates keep the steps apart)
                b.add("Toffoli", w, ((w + 3) % n, (w + 7) % n))
                b.add("Ry", w, (), param=r.uniform(-0.2, 0.2))
                b.add("Toffoli", w, ((w + 2) % n, (w + 5) % n))
        for w in range(n):
            b.add("CNot", (w + 1) % n, (w,))
    return b.build()


@pytest.mark.parametrize("kind", ["real", "complex", "phase", "grown"])
def test_custom_gates_keep_their_scaling(oracle, kind):
    """What a Custom matrix is off a unitary one belongs to the gate: 240 of them scale amplitudes by 1 -
    1.6e-11 and more, which is not taken for the rounding of library gates."""
    prof = _check(oracle, _chain(kind, 12, 20), nat.QGPU_C128)
    assert any(k.startswith("k_wide") for k in prof), prof


@pytest.mark.parametrize("precision", [nat.QGPU_C128, nat.QGPU_C64])
@pytest.mark.parametrize("n", [3, 4, 5, 6, 7, 10, 11, 12, 15])
def test_transform_rows_around_the_lines(oracle, n, precision):
    """Fourier transforms of a product state, between other layers, where their rows change between
    wide and tile passes (11 qubits of complex128; two phase tables in a row of complex64)."""
    b = ProgramBuilder(n)
    for w in range(n):
        b.add("Ry", w, (), param=0.3 + w)
    for i in range(n):
        b.add("H", i)
        for k in range(2, n - i + 1):
            b.add("CRk", i, (i + k - 1,), k=k)
    for i in range(n // 2):
        b.add("Swap", i, (n - 1 - i,))
    for w in range(n):
        b.add("Rx", w, (), param=0.2 * w - 1.0)
        b.add("CNot", (w + 1) % n, (w,))
    _check(oracle, b.build(), precision)
