"""How the marching kernels cut their columns (similie_b200/csrc/run_plan.cuh): the cut that the search over every
number of runs finds, from at most ten candidates a launch."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_the_cheapest_cut_from_a_few_candidates(tmp_path):
    exe = str(tmp_path / "run_plan")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror",
                           os.path.join(ROOT, "tests", "cpp", "run_plan.cpp"), "-o", exe])
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout.strip() == "runs ok", run.stdout + run.stderr
