"""Rounding to fixed point (csrc/spc_math.h) outside the range of the usual values,
on the CPU: values that are not finite or too large are marked, all others are
llrint's."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_out_of_range_values_are_marked(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "fixed_limits")
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-Werror", "-o", exe,
                    os.path.join(ROOT, "tests", "host", "fixed_limits.cpp"),
                    "-I", os.path.join(ROOT, "spc2_langevin_integration_gb300", "csrc")],
                   check=True, timeout=300)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.endswith("ok\n"), out.stdout + out.stderr
