"""Builds tests/cpp/packed_check.cu with nvcc for sm_103a and runs it: the packed f32x2 double-word operations
and the IEEE candidate screen must give the bits of the scalar operations (26M operand pairs)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu


def test_packed_operations_are_the_scalar_ones(tmp_path):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "packed_check")
    src = os.path.join(ROOT, "tests", "cpp", "packed_check.cu")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-o", exe, src],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr + r.stdout
