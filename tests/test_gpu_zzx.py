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
