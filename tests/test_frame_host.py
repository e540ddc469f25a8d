"""The frame of a run's undo (pauli_frame, quantr_gb300/csrc/plan.cpp) for angles down to the smallest
number. Bar: 2e-15, ten roundings of a complex product."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_frames_of_every_angle(tmp_path):
    exe = tmp_path / "frame_host"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(ROOT / "include"),
                        str(ROOT / "tests" / "cpp" / "frame_host.cpp"),
                        str(ROOT / "quantr_gb300" / "csrc" / "plan.cpp"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    assert float(r.stdout) <= 2e-15, r.stdout
