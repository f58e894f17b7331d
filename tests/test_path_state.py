"""The wavefront's path state after allocations that failed, on the CPU: path_state.cpp gives it a device
that refuses the k-th allocation."""
import os
import subprocess
from pathlib import Path


def test_path_state_survives_failed_allocations(tmp_path):
    src = Path(__file__).resolve().parent / "path_state.cpp"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = tmp_path / "path_state"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", f"{cuda}/include", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout
