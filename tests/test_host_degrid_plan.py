"""The degridder's chunk rule (fpga_gridding_b200/csrc/degrid_plan.h), compiled
with the host C++ compiler: its bounds, and its choice against the measured
times of every chunk length."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "fpga_gridding_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_degrid_chunk(tmp_path):
    exe = str(tmp_path / "degrid_plan_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC,
                    os.path.join(HERE, "degrid_plan_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip() == "ok"
