"""A task beside its maker (idx2_b200/csrc/parallel.h side_task, the device packer's compression of the
exponents): what it throws is thrown to the waiter instead of ending the process
(tests/cpp/side_task_check.cpp)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_side_task():
    build = os.path.join(HERE, "_build")
    os.makedirs(build, exist_ok=True)
    exe = os.path.join(build, "side_task_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I" + os.path.join(ROOT, "idx2_b200", "csrc"),
                    os.path.join(HERE, "cpp", "side_task_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
