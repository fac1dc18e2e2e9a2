"""Copies between host and device memory (idx2_b200/csrc/host_copy.h) over a fake CUDA runtime
(tests/cpp/host_copy_check.cpp): which memory goes through the threads, what they share with other
users of the context, and what a failing call leaves behind."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def check():
    build = os.path.join(HERE, "_build")
    os.makedirs(build, exist_ok=True)
    exe = os.path.join(build, "host_copy_check")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I" + os.path.join(ROOT, "idx2_b200", "csrc"),
                    "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(cuda, "include"),
                    os.path.join(HERE, "cpp", "host_copy_check.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("case", ["registered", "events", "failures"])
def test_host_copy(check, case):
    r = subprocess.run([check, case], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
