"""k_sample with one and with several shots per warp, in and out of order, against a running sum on
the host: chunks below and above a warp's width, several chunks, zero amplitudes, and uniforms past
the total (None).

A uniform within 1e-12 of a running sum may fall on either side (the sums' order differs); all other
indices are equal.
"""
import numpy as np
import pytest

from quantr_gb300 import _native as nat

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _lib(gpu_lib):
    yield


# 152 SMs x 16 warps: one shot per warp up to 4863 shots, two from 4864 on, 32 from 77824 on
@pytest.mark.parametrize("precision", [nat.QGPU_C128, nat.QGPU_C64])
@pytest.mark.parametrize("n,shots", [(1, 3), (3, 40), (5, 1000), (8, 4863), (9, 4864), (10, 7300), (13, 20001),
                                     (16, 77824), (6, 100003)])
def test_indices(n, shots, precision):
    r = np.random.default_rng(100 * n + shots)
    psi = r.standard_normal(1 << n) + 1j * r.standard_normal(1 << n)
    psi[r.random(1 << n) < 0.3] = 0
    psi[0] = 1
    psi /= np.linalg.norm(psi)
    if precision == nat.QGPU_C64:
        psi = psi.astype(np.complex64).astype(np.complex128)
    h = nat.Handle(n, precision)
    h.upload(psi)
    cum = np.cumsum(psi.real ** 2 + psi.imag ** 2)
    for u in (np.sort(r.random(shots)), r.random(shots)):
        u = u.copy()
        u[-1] = 1.5
        want = np.searchsorted(cum, u, side="right").astype(np.int64)
        want[want == 1 << n] = -1
        got = h.measure_uniforms(u)
        at = np.searchsorted(cum, u)
        near = np.minimum(np.abs(cum[np.minimum(at, cum.size - 1)] - u), np.abs(cum[np.maximum(at - 1, 0)] - u))
        ok = near > 1e-12
        assert np.array_equal(got[ok], want[ok])
