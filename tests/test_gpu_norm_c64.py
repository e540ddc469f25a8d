"""The norm of complex64 registers: packed f32 with error-free products and sums from 16 qubits
(k_norm_f32), f64 below. Both are sums in about f64 precision of the f32 amplitudes' squares:
relative error against numpy's f64 sum at most 1e-13 (numpy's pairwise sum itself: ~1e-15); scales whose
squares leave the f32 range take the f64 kernel."""
import numpy as np
import pytest

from quantr_gb300 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 4, 15, 16, 17, 21, 22])
@pytest.mark.parametrize("scale", [1.0, 1e-6, 1e6, 1e-25, 1e25])
def test_norm(gpu_lib, n, scale):
    r = np.random.default_rng(n)
    psi = (r.standard_normal(1 << n) + 1j * r.standard_normal(1 << n)).astype(np.complex64)
    psi *= np.float32(scale)
    h = nat.Handle(n, nat.QGPU_C64)
    h.upload(psi.astype(np.complex128))
    ref = float(np.sum(psi.real.astype(np.float64) ** 2 + psi.imag.astype(np.float64) ** 2))
    assert abs(h.norm() - ref) <= 1e-13 * ref


def test_norm_of_infinite_and_nan_amplitudes(gpu_lib):
    for bad in (np.inf, np.nan):
        psi = np.zeros(1 << 17, np.complex128)
        psi[12345] = bad
        h = nat.Handle(17, nat.QGPU_C64)
        h.upload(psi)
        assert not np.isfinite(h.norm())


@pytest.mark.parametrize("n", [16, 17, 20, 24])
def test_norm_of_equal_amplitudes(gpu_lib, n):
    """Equal amplitudes make equal rounding errors in every chunk: nothing cancels over the register.
    Bar: the squares are exact and a thread's 32 of them are summed to 2^-60, then f64 sums of at
    most 2 chunks per thread, 8 and 5 + 8 levels of a tree, 2^-53 each: 23 * 2^-53 < 4e-15."""
    r = np.random.default_rng(n)
    for c in r.uniform(0.5, 1.0, 4 if n == 24 else 16):
        v = np.float32(c * 2.0 ** (-n / 2))
        h = nat.Handle(n, nat.QGPU_C64)
        h.upload(np.full(1 << n, complex(float(v), 0.0)))
        assert abs(h.norm() / (float(v) ** 2 * 2.0 ** n) - 1.0) <= 4e-15
        h.close()
