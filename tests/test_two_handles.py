"""Handles used from different threads at once, whose launches of one kernel
differ in shape (and so in shared memory): no call may be refused or wrong.
(tests/cpp/two_handles_main.cpp; a program of its own, free of the interpreter lock.)"""
import os
import shutil
import subprocess

import pytest

import sbfs

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "two_handles_main.cpp")


@pytest.mark.parametrize("kernel", ["lane", "pool"])
def test_threads_with_launches_of_different_shapes(tmp_path, kernel):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if shutil.which("g++") is None:
        pytest.skip("g++ is not installed")
    exe = str(tmp_path / "two_handles_main")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", os.path.join(ROOT, "include"), SRC, "-o", exe,
                    sbfs.LIB_PATH, f"-Wl,-rpath,{os.path.dirname(sbfs.LIB_PATH)}"],
                   check=True, capture_output=True, text=True)
    out = subprocess.run([exe, kernel], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
