"""The elementary functions of csrc/spc_math.h compiled for the GPU: the root
against long double over squares of distances and radii (2^-900 to 2^900), the
logarithm's bound, and sine, cosine and logarithm bit for bit as on the CPU,
where they are compared with the C library's."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_functions_as_the_gpu_runs_them(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "math_device")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a", "-Xcompiler",
                    "-ffp-contract=off", "-o", exe, os.path.join(ROOT, "tests", "host", "math_device.cu"),
                    os.path.join(ROOT, "tests", "host", "math_host.cpp"), "-I", os.path.join(ROOT, "spc2_langevin_integration_gb300", "csrc")],
                   check=True, timeout=300)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0 and out.stdout.endswith("ok\n"), out.stdout + out.stderr
