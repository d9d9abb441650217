"""The flight kernels' tuning defines: every block size they document gets
through the compiler's checks (no GPU and no code generation needed)."""
import os
import shutil
import subprocess

import pytest

PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "c-mc_electron_b200")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="no nvcc")
@pytest.mark.parametrize("threads", [32, 128, 192, 256, 512])
def test_flight_threads(threads, tmp_path):
    r = subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-fdevice-syntax-only",
                        f"-DMCB200_FLIGHT_THREADS={threads}", "-I../include", "-Icsrc", "-c",
                        "csrc/flight_kernels.cu", "-o", str(tmp_path / "flight.o")], cwd=PKG, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
