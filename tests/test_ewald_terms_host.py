"""The FP64 Ewald terms against long double, checked on the host by
tests/host/ewald_terms.cu; needs nvcc, no GPU.
"""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_ewald_terms_on_host(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "ewald_terms")
    build = subprocess.run([nvcc, "-std=c++17", "-O2", "-gencode", "arch=compute_103a,code=sm_103a",
                            "-I" + os.path.join(ROOT, "include"),
                            os.path.join(HERE, "host", "ewald_terms.cu"), "-o", exe], capture_output=True, text=True)
    assert build.returncode == 0, build.stderr[-4000:]
    run = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    print(run.stdout)
    assert run.returncode == 0 and run.stdout.strip().endswith("OK"), run.stdout[-4000:]
