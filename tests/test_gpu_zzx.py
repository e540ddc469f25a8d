"""The tiled H psi / energy kernels (quantr_gb300/csrc/zzx.cu) against numpy in f64.

Tolerances, in units of S = sum|a| + sum|b| times <psi|psi>: complex128 sums float pairs (relative
error of a term at most 2^-46, so at most 2^-46 S over all terms): 1e-13 S. complex64 states round
each of the n + 1 terms of (H psi)[x] to f32 (relative 2^-24 each, at most 2^-24 (n + 2) S): 2e-6 S
for n <= 23.
"""
import numpy as np
import pytest

from quantr_gb300 import _native as nat
from quantr_gb300 import gradients as GR
from quantr_gb300 import workloads as W
from quantr_gb300.program import ProgramBuilder

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _lib(gpu_lib):
    yield


def _state(n, seed):
    r = np.random.default_rng(seed)
    psi = r.standard_normal(1 << n) + 1j * r.standard_normal(1 << n)
    return psi / np.linalg.norm(psi)


# 16: the plain kernel; 17: one later pass whose field reaches back over done bits; 19: the last
# size of two passes; 20: the first of three
@pytest.mark.parametrize("n", [16, 17, 19, 20])
@pytest.mark.parametrize("precision", [nat.QGPU_C128, nat.QGPU_C64])
def test_energy_against_numpy(n, precision):
    r = np.random.default_rng(n)
    a, b = r.standard_normal(n), r.standard_normal(n)
    psi = _state(n, 100 + n)
    if precision == nat.QGPU_C64:
        psi = psi.astype(np.complex64).astype(np.complex128)
    h = nat.Handle(n, precision)
    h.upload(psi)
    s = np.abs(a).sum() + np.abs(b).sum()
    tol = 1e-13 * s if precision == nat.QGPU_C128 else 2e-6 * s
    assert abs(h.expectation_zzx(a, b) - W.energy_dense(psi, a, b)) <= tol
    for i in (0, n // 2, n - 1):  # each kind of term alone, at both ends of the ring
        one = np.zeros(n)
        one[i] = 1.0
        zero = np.zeros(n)
        for aa, bb in ((one, zero), (zero, one)):
            assert abs(h.expectation_zzx(aa, bb) - W.energy_dense(psi, aa, bb)) <= tol / s
    assert np.array_equal(h.download(), psi)


@pytest.mark.parametrize("scale", [1e-30, 1e-12, 1e12, 1e40])
def test_energy_of_registers_outside_the_float_range(scale):
    """Squares of these amplitudes leave the float pairs' range (or come near it): the plain
    kernel's f64 result is returned."""
    n = 17
    r = np.random.default_rng(3)
    a, b = r.standard_normal(n), r.standard_normal(n)
    psi = _state(n, 5)
    h = nat.Handle(n)
    h.upload(psi * scale)
    ref = W.energy_dense(psi, a, b) * scale ** 2
    assert abs(h.expectation_zzx(a, b) - ref) <= 1e-13 * (np.abs(a).sum() + np.abs(b).sum()) * scale ** 2


def test_energy_reports_non_finite_registers():
    n = 17
    psi = _state(n, 6)
    psi[77] = np.nan
    h = nat.Handle(n)
    h.upload(psi)
    assert np.isnan(h.expectation_zzx(np.ones(n), np.ones(n)))


@pytest.mark.parametrize("n", [17, 20])
@pytest.mark.parametrize("precision", [nat.QGPU_C128, nat.QGPU_C64])
def test_gradient_through_the_tiled_vectors(n, precision):
    """phi and lambda written by the tiled kernels, against the plain f64 sweep
    (QGPU_MODE_F64). complex64 tolerance: the adjoint tests' 1e-4."""
    an = W.ansatz(n=n, layers=1, seed=9)
    prog = an.program()
    e, g = GR.energy_and_gradient(nat.Handle(n, precision), prog, an.a, an.b)
    re, rg = GR.energy_and_gradient(nat.Handle(n, nat.QGPU_C128, nat.QGPU_MODE_F64), prog, an.a, an.b)
    tol = 1e-11 if precision == nat.QGPU_C128 else 1e-4
    assert abs(e - re) <= tol
    assert np.max(np.abs(g - rg)) <= tol


# 17, 20: k_zzx of an energy; 22, 25, 27: k_zzx_energy, one, 54 and 216 tiles a CTA
@pytest.mark.parametrize("n", [17, 20, 22, 25, 27])
@pytest.mark.parametrize("precision", [nat.QGPU_C128, nat.QGPU_C64])
def test_energy_of_registers_with_few_values(n, precision):
    """Amplitudes that depend on the last two wires alone: every thread adds up equal terms, whose
    rounding errors do not cancel. Bar: of a term, the amplitudes' splits (2 * 2^-49), the product
    of their low parts (2^-48), and the errors of a tile's up to 8 sums (8 * 2^-24 * 2^-25), then sums
    over the tiles in triples of floats: 4e-14 of it (complex64: the tile's sums alone, of amplitudes
    and neighbours that are exact with one coefficient of 1)."""
    r = np.random.default_rng(n)
    for _ in range(3 if n < 25 else 1):
        c = r.uniform(0.3, 1.0, 4) * 2.0 ** (-n / 2)
        if precision == nat.QGPU_C64:
            c = c.astype(np.float32).astype(np.float64)
        h = nat.Handle(n, precision)
        psi = np.empty((1 << (n - 2), 4), np.complex128)
        psi[:] = c
        h.upload(psi.reshape(-1))
        del psi
        sq = c * c
        N = 2.0 ** (n - 2)
        one, zero = np.zeros(n), np.zeros(n)
        for wire in (0, n // 2, n - 3):  # X on a wire in |+>: the norm
            one[:] = 0.0
            one[wire] = 1.0
            want = N * sq.sum()
            assert abs(h.expectation_zzx(zero, one) - want) <= 4e-14 * want
        one[:] = 0.0
        one[n - 1] = 1.0
        want = 2.0 * N * (c[0] * c[1] + c[2] * c[3])
        assert abs(h.expectation_zzx(zero, one) - want) <= 4e-14 * want
        one[:] = 0.0
        one[n - 2] = 1.0  # ZZ of the last two wires
        want = N * (sq[0] - sq[1] - sq[2] + sq[3])
        assert abs(h.expectation_zzx(one, zero) - want) <= 4e-14 * N * sq.sum()
        h.close()


@pytest.mark.parametrize("n", [20, 25])
def test_gradient_energy_of_registers_with_few_values(n):
    """The same through H psi (energy_and_gradient): |+> on all wires and one Ry, whose energy is known;
    divided by the register's norm, the state's own rounding leaves 2^-48 per gate and wire."""
    b = ProgramBuilder(n)
    for w in range(n):
        b.add("H", w)
    b.add("Ry", n - 1, (), param=0.3)
    prog = b.build()
    h = nat.Handle(n)
    x = np.random.default_rng(n).uniform(0.5, 1.0, n)
    e, _ = GR.energy_and_gradient(h, prog, np.zeros(n), x)
    want = x[:-1].sum() + x[-1] * np.cos(0.3)
    assert abs(e / h.norm() - want) <= 1e-13 * x.sum()
