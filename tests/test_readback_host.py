"""The read-back code (csrc/mpm_readback.h) on the CPU, with the CUDA runtime's calls done on host memory and counted
(tests/host/fake_cudart.h)."""
import subprocess
from pathlib import Path

import pytest

from mpm_snow_sim2d_b200.build import CSRC, nvcc_path

HOST = Path(__file__).resolve().parent / "host"
CUDA_INCLUDE = Path(nvcc_path()).resolve().parents[1] / "include"


@pytest.mark.parametrize("name", ["readback_waits", "readback_ring"])
def test_readback(tmp_path, name):
    exe = tmp_path / name
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(HOST), "-I", str(CSRC), "-I", str(CUDA_INCLUDE),
                    str(HOST / f"{name}.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
