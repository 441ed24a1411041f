"""The plan of the one-launch triangular sweeps (csrc/sweep_plan.cpp), run on
the CPU the way the kernel walks it: a small driver compiled with g++ checks
on random, grid, chain and dense patterns that every row is swept once, that
every value a row uses has reached its CTA from an earlier level, that the
bytes announced per level are the bytes sent, and that the results equal a
row-by-row sweep; levels past the window and rows past a round are refused."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ngsolve-sparsesolv_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_sweep_plan_walk_equals_row_by_row():
    out = os.path.join(ROOT, "tests", "host", "_build")
    os.makedirs(out, exist_ok=True)
    exe = os.path.join(out, "sweep_plan_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, os.path.join(ROOT, "tests", "host", "sweep_plan_check.cpp"),
                    os.path.join(CSRC, "sweep_plan.cpp"), os.path.join(CSRC, "host_order.cpp"), "-o", exe], check=True,
                   timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert r.stdout.strip() == "ok"
