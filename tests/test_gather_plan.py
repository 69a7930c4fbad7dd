"""The node gather's runs of hexes (snac_b200/csrc/snac_gather_plan.h), compiled
on the host with tests/gather_plan_check.cpp: every hex a node takes terms from is
among those its block fetches, and a stage has room for them (no GPU needed)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_every_node_finds_its_hexes(tmp_path):
    exe = tmp_path / "gather_plan_check"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "snac_b200", "csrc"),
                    os.path.join(ROOT, "tests", "gather_plan_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("ok "), r.stdout
