"""run_steps_any (aloha_gb300/csrc/steps.h), the march's jump over a run of
skipped samples for step sizes that are not multiples of t's spacing, equals
the loop it replaces, bit for bit (tests/cpp/any_steps_check.cpp, the header
the kernels use compiled for the host)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_jump_equals_loop_for_any_step(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "any_steps_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(ROOT, "aloha_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "any_steps_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stdout + out.stderr
    assert " mismatches 0" in out.stdout
