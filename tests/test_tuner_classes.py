"""Classes of the merged-set autotuner: the times of sets that run one grid
whatever the candidate (one chunk per block) do not decide for larger sets, for
any number of lanes.  Built from the library's own tuner.h with g++; no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_fixed_grids_have_classes_of_their_own(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not found")
    exe = str(tmp_path / "tuner_classes_check")
    subprocess.run(["g++", "-std=c++17", "-O1", os.path.join(ROOT, "tests", "cpp", "tuner_classes_check.cpp"),
                    "-o", exe], check=True)
    out = subprocess.run([exe], stdout=subprocess.PIPE, text=True)
    assert out.returncode == 0 and out.stdout.strip().endswith("OK"), out.stdout
