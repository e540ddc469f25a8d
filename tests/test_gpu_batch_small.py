"""Circuits in shared memory (k_batch_small) and circuits that share one worker's handle, against
one adjoint sweep per circuit: every size up to the edges of the CTA forms, runs that need every sum
and both diagonals, index maps, and each multi-wire gate.

Tolerances: the batch tests' bars, complex128 1e-10 and complex64 1e-4.
"""
import numpy as np
import pytest

from quantr_gb300 import _native as nat
from quantr_gb300 import batch as B
from quantr_gb300 import gradients as GR
from quantr_gb300.program import ProgramBuilder

pytestmark = pytest.mark.gpu

ONE = ["Ry", "Rz", "H", "Phase", "X", "Rx", "T", "Y", "S", "X90", "Z", "Tdag"]
TWO = ["CNot", "Swap", "CZ", "CNot", "CY", "CR", "CRk"]


@pytest.fixture(autouse=True)
def _lib(gpu_lib):
    yield


def _circuit(n, seed):
    """Layers of random single-wire gates, then a CNot ring, single other gates, or a CNot / Swap run."""
    r = np.random.default_rng(seed)
    b = ProgramBuilder(n)
    for layer in range(4):
        for w in range(n):
            for g in r.choice(ONE, size=r.integers(0, 4)):
                b.add(str(g), w, (), param=r.uniform(-3, 3) if g in ("Rx", "Ry", "Rz", "Phase") else 0.0)
        if n > 1 and layer == 0:
            for w in range(n):
                b.add("CNot", (w + 1) % n, (w,))
        elif n > 1 and layer == 1:
            for g in TWO:
                c, t = r.choice(n, size=2, replace=False)
                kw = {"param": 0.7} if g == "CR" else {"k": 3} if g == "CRk" else {}
                b.add(g, int(t), (int(c),), **kw)
            if n > 2:
                c, d, t = r.choice(n, size=3, replace=False)
                b.add("Toffoli", int(t), (int(c), int(d)))
        elif n > 1:
            for g in ("CNot", "Swap", "CNot"):
                c, t = r.choice(n, size=2, replace=False)
                b.add(g, int(t), (int(c),))
    return B.BatchCircuit(b.build(), r.standard_normal(n), r.standard_normal(n))


@pytest.mark.parametrize("precision", [nat.QGPU_C128, nat.QGPU_C64])
@pytest.mark.parametrize("sizes", [(1, 2, 3, 4, 5, 6, 7, 8), (9, 10, 11, 12, 13), (14, 11, 17, 10, 15, 1),
                                   (13,), (6, 6)])
def test_batch_matches_per_circuit(sizes, precision):
    cs = [_circuit(n, 100 * n + k) for n in sizes for k in range(3)]
    e, g, _ = B.run_batch(cs, precision=precision)
    tol = 1e-10 if precision == nat.QGPU_C128 else 1e-4
    for i, c in enumerate(cs):
        h = nat.Handle(c.n)
        re, rg = GR.energy_and_gradient(h, c.program, c.a, c.b)
        h.close()
        assert abs(e[i] - re) <= tol, (c.n, i)
        assert np.max(np.abs(g[i] - rg), initial=0.0) <= tol, (c.n, i)

