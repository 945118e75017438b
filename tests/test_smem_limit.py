"""The dynamic shared memory limit of a kernel is per device: a second device's
first launch sets its own.  Checked on the host against a stand-in for the CUDA
runtime, and that no launcher sets the limit by itself."""
import os
import re
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "diamond-rust_b200", "csrc")


def test_limit_per_kernel_and_device(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    exe = str(tmp_path / "smem_limit_check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", os.path.join(ROOT, "include"), "-I",
                        cuda, os.path.join(ROOT, "tests", "smem_limit_check.cpp"), "-o", exe], capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


def test_launchers_share_it():
    for name in os.listdir(CSRC):
        path = os.path.join(CSRC, name)
        if os.path.isfile(path) and name != "smem_limit.h":
            assert not re.search(r"cudaFuncSetAttribute|static \w+ configured", open(path).read()), name
