"""Range profiles and device memory, without a GPU: the engine's host code on a fake of the CUDA runtime
(tests/cpp/no_memory.cpp) whose allocations fail as they do when another user of the device took
the memory. Every call that the direct kernels can serve is served."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_calls_are_served_where_the_table_cannot_be_allocated(tmp_path):
    exe = tmp_path / "no_memory"
    pkg = ROOT / "sarlab-tdc_gb300"
    cmd = ["g++", "-std=c++17", "-O1", "-I", str(ROOT / "include"), "-I", str(pkg / "csrc"), "-I",
           "/usr/local/cuda/include", str(ROOT / "tests" / "cpp" / "no_memory.cpp"), str(pkg / "csrc" / "tdc_capi.cpp"),
           "-lpthread", "-ldl", "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
