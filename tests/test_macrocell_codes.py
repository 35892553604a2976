"""The macrocell codes: their passes equal the definition of a cell's reach
(tests/cpp/reach_check.cpp, the header the kernels use compiled for the host)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_passes_equal_the_definition(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "reach_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "aloha_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "reach_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
