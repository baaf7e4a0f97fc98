"""CPU: a chain tuning that fails leaves the table's entry as it was, a
caller's setting as well as the default."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_entry_survives_a_failed_tuning(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    exe = str(tmp_path / "chain_tune_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "latttmat_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "chain_tune_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], env=dict(os.environ, CUDA_VISIBLE_DEVICES=""), capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
