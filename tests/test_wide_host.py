"""Wide passes of the planner (quantr_gb300/csrc/plan.cpp, wide_schedule) on the host: every step of
the scheduled passes applied in order in complex128 (tests/cpp/wide_emulator.cpp) against the
oracle. Bar: 1e-12, the planner tests' (gate matrices are multiplied and split, not applied
one by one)."""
import os
import subprocess
from pathlib import Path

import numpy as np
import pytest

from quantr_gb300 import workloads as W
from quantr_gb300.program import ProgramBuilder

ROOT = Path(__file__).resolve().parent.parent
TOL = 1e-12


@pytest.fixture(scope="module")
def emulator(tmp_path_factory):
    exe = tmp_path_factory.mktemp("wide") / "wide_emulator"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(ROOT / "include"),
                        str(ROOT / "tests" / "cpp" / "wide_emulator.cpp"),
                        str(ROOT / "quantr_gb300" / "csrc" / "plan.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


def _run(emulator, prog, tmp_path, bits, regs, low, pairs, pair_fusion=1):
    f = {k: tmp_path / f"{k}.bin" for k in ("ops", "mats", "none", "out")}
    np.ascontiguousarray(prog.ops).tofile(f["ops"])
    np.ascontiguousarray(prog.mats, dtype=np.float64).tofile(f["mats"])
    np.ascontiguousarray(prog.none, dtype=np.uint8).tofile(f["none"])
    env = dict(os.environ, WIDE_BITS=str(bits), WIDE_REGS=str(regs), WIDE_LOW=str(low),
               WIDE_PAIRS=str(pairs))
    r = subprocess.run([str(emulator), str(prog.n), str(f["ops"]), str(f["mats"]), str(f["none"]),
                        str(f["out"]), str(pair_fusion), "280", "2", "0", "1"],
                       capture_output=True, text=True, timeout=300, env=env)
    assert r.returncode == 0, r.stderr
    counts = dict(zip(r.stdout.split()[::2], map(int, r.stdout.split()[1::2])))
    return np.fromfile(f["out"], dtype=np.complex128), counts


def _everything(n, seed):
    """Every gate kind, Custom gates (dense, damped, with None columns), long runs of each."""
    r = np.random.default_rng(seed)
    b = ProgramBuilder(n)
    one = ["H", "X", "Y", "Z", "S", "Sdag", "T", "Tdag", "X90", "Y90", "MX90", "MY90"]
    for _ in range(4):
        for w in range(n):
            k = r.integers(16)
            if k < 12:
                b.add(one[k], w)
            else:
                b.add(["Rx", "Ry", "Rz", "Phase"][k - 12], w, (), param=r.uniform(-6, 6))
        for _ in range(n):
            p = [int(x) for x in r.permutation(n)[:3]]
            k = r.integers(8)
            if k == 0:
                b.add("Toffoli", p[0], (p[1], p[2]))
            elif k == 1:
                b.add("CR", p[0], (p[1],), param=r.uniform(-3, 3))
            elif k == 2:
                b.add("CRk", p[0], (p[1],), k=int(r.integers(1, 6)))
            else:
                b.add(["CZ", "CY", "CNot", "Swap", "CNot"][k - 3], p[0], (p[1],))
        m = r.standard_normal((2, 2)) + 1j * r.standard_normal((2, 2))
        b.add_custom(int(r.integers(n)), [], m / np.linalg.norm(m), np.zeros(2, np.uint8))
        p = [int(x) for x in r.permutation(n)[:2]]
        cu = np.eye(4, dtype=complex)
        cu[2:, 2:] = np.linalg.qr(r.standard_normal((2, 2)) + 1j * r.standard_normal((2, 2)))[0].T
        b.add_custom(p[0], [p[1]], cu, np.zeros(4, np.uint8))
        none = np.zeros(4, np.uint8)
        none[int(r.integers(4))] = 1
        b.add_custom(p[1], [p[0]], r.standard_normal((4, 4)) / 2, none)
    return b.build()


# tile and round widths of the complex128 and complex64 kernels, and narrow ones
@pytest.mark.parametrize("bits,regs,low,pairs", [(10, 3, 2, 0), (12, 4, 3, 0), (5, 2, 2, 6), (4, 2, 0, 0),
                                                 (6, 4, 3, 0)])
@pytest.mark.parametrize("n", [2, 3, 7, 10, 12])
def test_every_gate_kind(emulator, oracle, tmp_path, n, bits, regs, low, pairs):
    if n < 3:
        b = ProgramBuilder(n)
        for w in range(n):
            b.add("Ry", w, (), param=0.3 + w)
            b.add("Rz", w, (), param=0.7)
        b.add("CNot", 1, (0,))
        b.add("Rx", 0, (), param=1.1)
        b.add("Swap", 0, (1,))
        prog = b.build()
    else:
        prog = _everything(n, 10 * n + bits)
    ref = oracle.simulate(prog, engine=oracle.DENSE)
    out, _ = _run(emulator, prog, tmp_path, bits, regs, low, pairs)
    assert np.max(np.abs(out - ref)) <= TOL


@pytest.mark.parametrize("family,n,bits,regs,low,most", [
    ("ansatz", 12, 10, 3, 2, 12), ("ansatz", 10, 10, 3, 2, 3), ("columns", 11, 10, 3, 2, 20),
    ("brickwork", 12, 8, 2, 2, 26), ("brickwork", 13, 12, 4, 3, 8)])
def test_families(emulator, oracle, tmp_path, family, n, bits, regs, low, most):
    """The workload families take fewer passes than there are layers of gates to reorder."""
    prog = {"ansatz": lambda: W.ansatz(n=n, layers=4, seed=1).program(),
            "columns": lambda: W.random_columns(n=n, columns=30, seed=2),
            "brickwork": lambda: W.brickwork_qft(n=n, layers=10, seed=3)}[family]()
    ref = oracle.simulate(prog, engine=oracle.DENSE)
    out, counts = _run(emulator, prog, tmp_path, bits, regs, low, 0)
    assert np.max(np.abs(out - ref)) <= TOL
    assert 1 <= counts["wide"] <= most, counts
