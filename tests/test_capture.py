"""Recording steps into a graph (snac_b200/csrc/snac_capture.h), compiled on the
host with tests/capture_check.cpp: a failure of any call leaves the stream out
of the capture, no graph, and the bookkeeping as it was (no GPU needed)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_a_failed_capture_leaves_nothing_behind(tmp_path):
    exe = tmp_path / "capture_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "snac_b200", "csrc"),
                    os.path.join(ROOT, "tests", "capture_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
