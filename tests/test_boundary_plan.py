"""The split of the four boundary sides into regions that run in one launch (host rule, on the CPU)."""
from __future__ import annotations

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_regions_equal_the_sides_in_order(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.run(["/usr/bin/g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "celeris_b200", "csrc"),
                    os.path.join(ROOT, "tests", "boundary_plan_check.cpp"), "-o", exe], check=True)
    planned, refused, wrong, races = map(int, subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split())
    assert planned > 10000 and refused > 10000   # both kinds of domain were met
    assert wrong == 0 and races == 0
