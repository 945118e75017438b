"""A call that fails between forking work to other streams and joining them
waits for those streams before it frees what they read.  The guard is checked on
the host against a stand-in; every fork of the pipeline uses it."""
import os
import re
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "diamond-rust_b200", "csrc")


def test_failed_call_waits_for_its_streams(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")
    exe = str(tmp_path / "stream_fork_check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", cuda,
                        os.path.join(ROOT, "tests", "stream_fork_check.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr


def test_forks_are_guarded():
    text = open(os.path.join(CSRC, "pipeline.cu")).read()
    for body in re.split(r"\n}\n", text):
        forks = re.search(r"cudaStreamWaitEvent\((?!c->stream)", body)
        if forks and "start_early_ref" not in body and "Search::filtered_seeds" not in body:
            guard = body.index("ForkGuard forked;")
            assert guard < body.index("forked.add(") < forks.start() < body.index("forked.joined();")
    # the side stream's early seeds: ~Search waits for them while early_ref is set
    early = text[text.index("void Search::start_early_ref() {"):]
    assert early.index("early_ref = true;") < early.index("filtered_seeds(")
