"""Host side of the kernel launches (csrc/pb_launch.cuh) on fakes of the
runtime's calls, compiled and run as a program of its own, without a GPU."""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")
NVCC = os.path.join(CUDA, "bin", "nvcc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not os.path.exists(NVCC):
        pytest.skip("needs nvcc")
    exe = str(tmp_path_factory.mktemp("launch") / "launch_state")
    cpp = os.path.join(ROOT, "tests", "cpp")
    cmd = [NVCC, "-std=c++17", "-cudart", "shared", "-gencode", "arch=compute_100a,code=sm_100a",
           "-I", os.path.join(ROOT, "pencil-rs_b200", "csrc"), os.path.join(cpp, "launch_state.cu"),
           os.path.join(cpp, "runtime_fakes.cpp"), "-o", exe, "-Xlinker", "-rpath=" + os.path.join(CUDA, "lib64")]
    proc = subprocess.run(cmd, capture_output=True, text=True)
    assert proc.returncode == 0, proc.stderr
    return exe


def test_launch_state(program):
    proc = subprocess.run([program], capture_output=True, text=True, timeout=60)
    assert proc.returncode == 0 and "launch ok" in proc.stdout, proc.stdout + proc.stderr
