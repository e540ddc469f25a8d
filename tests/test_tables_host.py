"""Phase tables of the planner (quantr_gb300/csrc/plan.cpp, fold_entries) on the host: runs of
diagonal gates near the unit circle (products in pairs of doubles) and with Custom factors that
reach 1e20 and 1e-20 (long double; no table entry leaves the range of double), applied to a uniform register by the plan emulator, against
products in long double. Bar: 4e-15 of each amplitude (12 Hadamard products, at most 8 roundings of
table entries and their products)."""
import os
import subprocess
from pathlib import Path

import numpy as np
import pytest

from quantr_gb300.program import ProgramBuilder

ROOT = Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("n,custom", [(2, 0.0), (7, 0.0), (12, 0.0), (12, 20.0), (5, 20.0)])
def test_table_products(tmp_path, n, custom):
    exe = tmp_path / "emulator"
    src = [str(ROOT / "tests" / "cpp" / "plan_emulator.cpp"), str(ROOT / "quantr_gb300" / "csrc" / "plan.cpp")]
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(ROOT / "include"),
                        *src, "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    rng = np.random.default_rng(n)
    b = ProgramBuilder(n)
    idx = np.arange(1 << n)
    bit = [((idx >> (n - 1 - w)) & 1).astype(bool) for w in range(n)]
    want = np.full(1 << n, 1, np.clongdouble) / np.sqrt(np.longdouble(2)) ** n
    for w in range(n):
        b.add("H", w)
    for k in range(3 * n):
        t, c = (int(x) for x in rng.permutation(n)[:2])
        a = rng.uniform(-3, 3)
        if k % 3 == 0:
            b.add("Rz", t, (), param=a)
            want *= np.where(bit[t], np.exp(0.5j * a), np.exp(-0.5j * a))
        elif k % 3 == 1 or not custom:
            b.add("CR", t, (c,), param=a)
            want *= np.where(bit[t] & bit[c], np.exp(1j * a), 1)
        else:  # large and small factors in turn
            d = 10.0 ** (custom if (k // 3) % 2 else -custom)
            b.add_custom(t, [], np.diag([1.0, d]).astype(np.complex128), np.zeros(2, np.uint8))
            want *= np.where(bit[t], np.longdouble(d), 1)
    p = b.build()
    f = {k: tmp_path / f"{k}.bin" for k in ("ops", "mats", "none", "out")}
    np.ascontiguousarray(p.ops).tofile(f["ops"])
    np.ascontiguousarray(p.mats, dtype=np.float64).tofile(f["mats"])
    np.ascontiguousarray(p.none, dtype=np.uint8).tofile(f["none"])
    r = subprocess.run([str(exe), str(n), *(str(f[k]) for k in ("ops", "mats", "none", "out")), "0", "280", "2",
                        "0", "1"], capture_output=True, text=True, timeout=300, env=dict(os.environ))
    assert r.returncode == 0, r.stderr
    got = np.fromfile(f["out"], dtype=np.complex128)
    ok = (np.abs(want) < 1e290) & (np.abs(want) > 1e-290)
    assert ok.sum() > 1
    assert np.max(np.abs(got - want)[ok] / np.abs(want)[ok]) <= 4e-15
