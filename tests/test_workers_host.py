"""The host threads of a batch (quantr_gb300/csrc/workers.h): each one takes over the caller's CUDA
device before it creates a handle."""
import re
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_threads_enter_before_their_work(tmp_path):
    exe = tmp_path / "workers_host"
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", str(ROOT / "tests" / "cpp" / "workers_host.cpp"),
                        "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "fails 0", r.stdout + r.stderr


def test_batches_start_threads_through_it_alone():
    """A std::thread of its own would create its handles on device 0."""
    text = (ROOT / "quantr_gb300" / "csrc" / "batch.cu").read_text()
    assert "std::thread" not in text
    assert re.search(r"auto enter = .*?cudaSetDevice\(dev\).*?run_workers\(workers, enter, work\)", text, re.S)
