"""The rule that chooses between one launch for all levels of a triangular sweep and
a launch per level (csrc/sweep_plan.cpp: SweepPlanHost::build with the other way's
time, level_launches_us), on patterns whose both times were measured: wide, few or
scattered levels keep their launches."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ngsolve-sparsesolv_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_the_rule_picks_the_faster_way():
    out = os.path.join(ROOT, "tests", "host", "_build")
    os.makedirs(out, exist_ok=True)
    exe = os.path.join(out, "sweep_rule_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, os.path.join(ROOT, "tests", "host", "sweep_rule_check.cpp"),
                    os.path.join(CSRC, "sweep_plan.cpp"), os.path.join(CSRC, "host_order.cpp"), "-o", exe], check=True,
                   timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert r.stdout.strip() == "ok"
