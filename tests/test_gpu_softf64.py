"""Builds tests/cpp/softf64_check.cu with nvcc for sm_103a and runs it: the integer-pipe division and
square root (pg_softf64.cuh) must give the bits of the device's IEEE operations on 268M operand pairs,
special values and operands next to rounding boundaries among them."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.gpu


def test_division_and_root_are_ieee(tmp_path):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path / "softf64_check")
    src = os.path.join(ROOT, "tests", "cpp", "softf64_check.cu")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-o", exe, src],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr + r.stdout
