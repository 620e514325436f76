"""FP64 multiplication, division and square root on the integer pipes
(csrc/rc_soft.cuh) against the hardware's, bit for bit: on the processor, and
on the GPU (needs a GB300 and nvcc)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "rocketcombustor_gb300", "csrc")
SRC = os.path.join(HERE, "cuda", "soft_check.cu")


def _check(cmd, exe, n):
    subprocess.run(cmd + [f"-I{CSRC}", f"-I{os.path.join(os.path.dirname(HERE), 'include')}", "-o", exe, SRC], check=True)
    r = subprocess.run([exe, str(n)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "mismatches 0" in r.stdout, r.stdout + r.stderr


def test_integer_fp64_equals_the_processors(tmp_path):
    _check(["g++", "-x", "c++", "-O2", "-ffp-contract=off", "-std=c++17"], str(tmp_path / "soft"), 1 << 22)


@pytest.mark.gpu
def test_integer_fp64_equals_the_gpus(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    _check([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-std=c++17"],
           str(tmp_path / "soft"), 1 << 28)
