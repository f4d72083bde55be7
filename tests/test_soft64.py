"""The integer FP64 division, square root, sine and cosine (csrc/soft64.cuh),
compiled for the host, against the machine's FP64."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    inc = "/usr/local/cuda/include"
    if not shutil.which("g++") or not os.path.exists(os.path.join(inc, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    out = str(tmp_path_factory.mktemp("soft64") / "check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", inc, "-I",
                    os.path.join(ROOT, "test_particle_gb300", "csrc"), os.path.join(ROOT, "tests", "soft64_check.cpp"),
                    "-o", out], check=True)
    return out


@pytest.mark.parametrize("family", range(5))
def test_division_root_and_trigonometry(program, family):
    r = subprocess.run([program, str(family), "400000"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
