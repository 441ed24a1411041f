"""The ring of stages of the one-launch triangular sweeps (SweepPlanHost::ring_stages),
against a model of its barriers: with copies that land late, a warp must never take an
older round for its own. Rings that are no multiple of the groups do (the model shows
it), so none is planned."""
from __future__ import annotations

import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "ngsolve-sparsesolv_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_every_warp_finds_its_round():
    out = os.path.join(ROOT, "tests", "host", "_build")
    os.makedirs(out, exist_ok=True)
    exe = os.path.join(out, "sweep_ring_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, os.path.join(ROOT, "tests", "host", "sweep_ring_check.cpp"),
                    "-o", exe], check=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-2000:] + r.stderr[-2000:]
    assert r.stdout.strip() == "ok"
