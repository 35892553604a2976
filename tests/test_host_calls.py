"""What the host side of the C ABI (aloha_gb300/csrc/api.cpp) leaves done when a
call returns, on a stand-in for the CUDA runtime that puts copies and kernels
off until their stream is waited for (tests/cpp/fake_cuda.h)."""
import os
import subprocess

import pytest

from aloha_gb300 import build as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    try:
        cc = B.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not found")
    exe = str(tmp_path_factory.mktemp("host_calls") / "check")
    subprocess.run([cc, "-O1", "-std=c++17", "-Xcompiler", "-ffp-contract=off", "-cudart", "none", "-I", B.CSRC,
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "tests", "cpp"),
                    os.path.join(ROOT, "tests", "cpp", "host_calls_check.cpp"), os.path.join(B.CSRC, "api.cpp"),
                    os.path.join(B.CSRC, "order.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("name", ["scene_flag", "table", "composite", "large", "views", "chunk_counters"])
def test_calls_leave_the_device_ready(check, name):
    out = subprocess.run([check, name], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
