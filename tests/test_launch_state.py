"""What the library keeps per kernel between launches (launch_state.cuh), on the host
with counted fakes (tests/cpp/test_launch_state.cu): limits belong to a device and a
kernel, only grow, and are safe with several threads; a kernel's cluster size is its
own, and none where the device holds no such cluster."""
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_launch_state_host(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = tmp_path / "test_launch_state"
    subprocess.run([nvcc, "-std=c++17", "-O2", "-Wno-deprecated-gpu-targets",
                    str(ROOT / "tests" / "cpp" / "test_launch_state.cu"),
                    "-o", str(exe), "-lpthread"], check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "launch state ok" in r.stdout
