"""The CUDA build: the same code from every build.  -split-compile cuts a
file among threads, and the cut, with it the registers of every kernel that
calls a function, changed from one build to the next."""
import glob
import os

from snac_b200 import build as B


def test_files_are_compiled_whole_and_apart(monkeypatch):
    monkeypatch.setattr(B, "nvcc", lambda: "nvcc")
    commands = B.compile_commands("/obj")
    files = sorted(glob.glob(os.path.join(B.CSRC, "*.cu")))
    assert [c[-1] for c in commands] == files and len(files) > 1
    for c in commands:
        assert not any(a.startswith(("-split-compile", "--split-compile", "-rdc", "-dc")) for a in c)
        assert "-fmad=false" in c
