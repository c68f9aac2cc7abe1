"""A training scratch or data set whose allocation failed is not used by the calls
that follow: mlp_trainer.cpp on a CUDA runtime that runs out of memory on request
(tests/trainer_allocation_check.cpp).  CPU only."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "wasl_b200", "csrc")
CXX = shutil.which("g++")
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
CUDA = os.path.join(os.path.dirname(os.path.dirname(NVCC)), "include")


def test_calls_after_a_failed_allocation(tmp_path):
    if CXX is None or not os.path.exists(os.path.join(CUDA, "cuda_runtime.h")):
        pytest.skip("no g++ or no CUDA headers")
    out = tmp_path / "check"
    subprocess.run([CXX, "-std=c++20", "-O1", "-g", f"-I{CSRC}", f"-I{CUDA}",
                    f"-I{os.path.join(ROOT, 'include')}",
                    os.path.join(ROOT, "tests", "trainer_allocation_check.cpp"),
                    os.path.join(CSRC, "mlp_trainer.cpp"), "-o", str(out), "-ldl"], check=True)
    run = subprocess.run([str(out)], capture_output=True, text=True)
    assert run.returncode == 0 and "0 failures" in run.stdout, run.stdout + run.stderr
