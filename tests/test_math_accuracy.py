"""The elementary functions of the per-particle work (csrc/spc_math.h) against
the C library's long double ones, on the CPU: over their ranges and at the
points and seams of their tables, and the rounding to fixed point bit for bit
against llrint."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_functions_are_within_their_bounds(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "math_accuracy")
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-Werror", "-o", exe,
                    os.path.join(ROOT, "tests", "host", "math_accuracy.cpp"),
                    "-I", os.path.join(ROOT, "spc2_langevin_integration_gb300", "csrc")],
                   check=True, timeout=300)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.endswith("ok\n"), out.stdout + out.stderr
