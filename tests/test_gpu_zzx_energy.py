"""Energies of complex128 registers taken pair by pair (k_zzx_energy in quantr_gb300/csrc/zzx.cu)
against numpy in f64, at its smallest size, with a last pass that reaches back over done bits, and
each kind of term alone.

Tolerance: the tiled kernels' tests', 1e-13 of sum|a| + sum|b|.
"""
import numpy as np
import pytest

from quantr_gb300 import _native as nat
from quantr_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _lib(gpu_lib):
    yield


@pytest.mark.parametrize("n", [22, 23])
def test_energy_by_pairs(n):
    r = np.random.default_rng(n)
    a, b = r.standard_normal(n), r.standard_normal(n)
    psi = r.standard_normal(1 << n) + 1j * r.standard_normal(1 << n)
    psi /= np.linalg.norm(psi)
    h = nat.Handle(n)
    h.upload(psi)
    s = np.abs(a).sum() + np.abs(b).sum()
    assert abs(h.expectation_zzx(a, b) - W.energy_dense(psi, a, b)) <= 1e-13 * s
    for i in (0, 3, 6, 9, n - 14, n - 7, n - 3, n - 1):  # a wire of every arrangement and pass
        one, zero = np.zeros(n), np.zeros(n)
        one[i] = 1.0
        assert abs(h.expectation_zzx(zero, one) - W.energy_dense(psi, zero, one)) <= 1e-13
    h.upload(1e25 * psi)  # squares outside the float pairs' range: the plain kernel's result
    want = W.energy_dense(1e25 * psi, a, b)
    assert abs(h.expectation_zzx(a, b) - want) <= 1e-13 * s * 1e50
