"""Streams for the groups of a set (icx_forks.h) with each creation of a stream
or event failing in turn, and with a piece of work that fails (CPU)."""
import os
import subprocess

from test_cpp_facade import CUDA_INC, ROOT, needs_gxx


@needs_gxx
def test_forks(tmp_path):
    exe = str(tmp_path / "forks_check")
    # the CUDA calls of the header's own Api are declared, never called: nothing to link
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-D_GLIBCXX_ASSERTIONS", "-I",
                        os.path.join(ROOT, "iceicle_b200", "csrc"), "-I", CUDA_INC,
                        os.path.join(ROOT, "tests", "cpp", "forks_check.cpp"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
