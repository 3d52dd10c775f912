"""Fields of D*D values a particle outgrow 2^31 values at 239M particles, which fit the GPU. What indexes them is 64 bits
wide: the structures the kernels take the particle count and the queue's capacity from, and what kernels read them into."""
import re
import subprocess

import pytest

from mpm_snow_sim2d_b200.build import CSRC, GENCODE, INCLUDE, nvcc_path


def test_counts_are_64_bit(tmp_path):
    src = tmp_path / "width.cu"
    src.write_text('#include "mpm_kernels.cuh"\n'
                   "static_assert(sizeof(mpm::Particles::n) == 8);\n"
                   "static_assert(sizeof(mpm::SlowQueue::capacity) == 8);\n")
    r = subprocess.run([nvcc_path(), *GENCODE, "-std=c++17", "--expt-relaxed-constexpr", "-I", str(INCLUDE), "-I", str(CSRC),
                        "-cuda", "-o", str(tmp_path / "width.ii"), str(src)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cuh")), ids=lambda p: p.name)
def test_kernels_do_not_narrow_them(path):
    narrow = re.findall(r"^.*\bint \w+ = (?:P\.n|Q\.capacity)\b.*$", path.read_text(), re.M)
    assert [s for s in narrow if "long long" not in s] == []
