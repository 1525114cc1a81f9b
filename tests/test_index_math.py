"""Index arithmetic of the kernels for the largest grids, compiled for the host and run under the compiler's
overflow sanitizer (tests/cpp/index_check.cu)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_largest_grids(tmp_path):
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "index_check")
    src = os.path.join(ROOT, "tests", "cpp", "index_check.cu")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17",
                        "-I", os.path.join(ROOT, "include"), "-Xcompiler",
                        "-fsanitize=signed-integer-overflow,-fno-sanitize-recover=signed-integer-overflow", "-o", exe,
                        src], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
