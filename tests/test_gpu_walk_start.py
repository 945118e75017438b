"""The traceback walk reports a best cell outside the matrix or the band as an
internal error.  No search makes one, so tests/walk_check.cu calls the walk."""
import os
import shutil
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_walk_reports_a_start_outside(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "walk_check")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-I",
                        os.path.join(ROOT, "diamond-rust_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                        os.path.join(ROOT, "tests", "walk_check.cu"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
