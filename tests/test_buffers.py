"""A solve set's state buffers after a failed device allocation: no room is
recorded for states that do not exist, and the next set-up allocates them.
Built from the library's own buffers.h with g++ over fake CUDA calls; no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_state_buffers_after_a_failed_allocation(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")
    if not shutil.which("g++") or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("g++ or the CUDA headers not found")
    exe = str(tmp_path / "buffers_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + cuda, os.path.join(ROOT, "tests", "cpp", "buffers_check.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], stdout=subprocess.PIPE, text=True)
    assert out.returncode == 0 and out.stdout.strip().endswith("OK"), out.stdout
