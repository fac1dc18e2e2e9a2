"""The kernels' shared-memory limits, raised once per context (idx2_b200/csrc/device.h): a failed call
is reported and tried again by the next decode (tests/cpp/smem_limits_check.cpp, a fake of the failing
call)."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_smem_limits_are_tried_again():
    build = os.path.join(HERE, "_build")
    os.makedirs(build, exist_ok=True)
    exe = os.path.join(build, "smem_limits_check")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I" + os.path.join(ROOT, "idx2_b200", "csrc"),
                    "-I" + os.path.join(ROOT, "include"), "-I" + os.path.join(cuda, "include"),
                    os.path.join(HERE, "cpp", "smem_limits_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
