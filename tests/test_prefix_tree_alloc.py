"""CPU: a prefix tree whose tables could not be allocated is no tree.

An operator may get its tree at its first gradient; a build that ran out of
memory must leave it without one, so that the next gradient builds it again.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_failed_build_leaves_no_tree(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("needs nvcc")
    exe = str(tmp_path / "prefix_tree_alloc_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "latttmat_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "prefix_tree_alloc_check.cu"), "-o", exe], check=True)
    env = dict(os.environ, CUDA_VISIBLE_DEVICES="")
    r = subprocess.run([exe], env=env, capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
