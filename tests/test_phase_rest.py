"""What rounding leaves of a phase's sine and cosine (csrc/spc_math.h), on the CPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rest_is_within_its_bound(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no g++")
    exe = str(tmp_path / "phase_rest")
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-Wall", "-Werror", "-o", exe,
                    os.path.join(ROOT, "tests", "host", "phase_rest.cpp"),
                    "-I", os.path.join(ROOT, "spc2_langevin_integration_gb300", "csrc")],
                   check=True, timeout=300)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.endswith("ok\n"), out.stdout + out.stderr
