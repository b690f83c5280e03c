"""The row arithmetic of the batched CG kernels (similie_b200/csrc/item_rows.cuh) at the end of the accepted range:
problems hold up to 2^31 - 1 unknowns, and a kernel looks a round of rows past its item's end."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_rows_stay_in_their_item(tmp_path):
    exe = str(tmp_path / "item_rows")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", "-fsanitize=undefined",
                           "-fno-sanitize=pointer-overflow,null", "-fno-sanitize-recover=all",
                           os.path.join(ROOT, "tests", "cpp", "item_rows.cpp"), "-o", exe])
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout.strip() == "rows ok", run.stdout + run.stderr


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_items_of_a_problem(tmp_path):
    """Whole nodes, at most one wave of CTAs, and enough of them (the divergence gauge had a quarter)."""
    exe = str(tmp_path / "item_step")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror",
                           os.path.join(ROOT, "tests", "cpp", "item_step.cpp"), "-o", exe])
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout.strip() == "items ok", run.stdout + run.stderr
