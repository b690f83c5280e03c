"""Solves of different sizes that run the same kernel instance, from several host threads at once.

What a launch allows its kernel (shared memory) belongs to the kernel and the device, not to the call, so no
call may take it away from another thread's between its setting and its launch.  The threads are native ones
(tests/cpp/solve_threads.cpp): the window is a few hundred nanoseconds, and with each call setting its own
need one call in 10,000 to 60,000 was refused.
"""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = "/usr/local/cuda"


# FP64 instances of two nodes a thread (24.7 and 46 KB) and of four (53 and 55 KB)
@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
@pytest.mark.parametrize("grids", [(5, 5, 900, 3), (161, 161, 256, 256)])
def test_sizes_of_one_instance_side_by_side(tmp_path, grids):
    lib = os.path.join(ROOT, "similie_b200", "libsil_b200.so")
    exe = str(tmp_path / "solve_threads")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-I", os.path.join(ROOT, "include"),
                           "-I", os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "cpp", "solve_threads.cpp"),
                           "-o", exe, lib, "-L", os.path.join(CUDA, "lib64"), "-lcudart", "-lpthread",
                           "-Wl,-rpath," + os.path.dirname(lib) + ":" + os.path.join(CUDA, "lib64")])
    out = subprocess.run([exe] + [str(g) for g in grids] + ["3", "8"], check=True, capture_output=True, text=True).stdout
    calls, _, errors, _ = out.split(maxsplit=3)
    assert int(calls) > 10000 and int(errors) == 0, out
