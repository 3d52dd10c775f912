"""mpm_batch_step after a call that failed half way, on the CPU: csrc/mpm_batch.cu against a CUDA runtime that runs nothing and
fails where it is told to (tests/host/batch_failures.cu, fake_cudart.cpp)."""
import subprocess
from pathlib import Path

from mpm_snow_sim2d_b200.build import CSRC, GENCODE, INCLUDE, nvcc_path

HOST = Path(__file__).resolve().parent / "host"


def test_calls_after_a_failed_one(tmp_path):
    exe = tmp_path / "batch_failures"
    subprocess.run([nvcc_path(), *GENCODE, "-std=c++17", "-O0", "-Xptxas", "-O0", "--expt-relaxed-constexpr", "-cudart", "none",
                    "-I", str(INCLUDE), "-I", str(CSRC), str(HOST / "batch_failures.cu"), str(HOST / "fake_cudart.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
