"""The pieces that the boundary corners are cut into (host rule, on the CPU)."""
from __future__ import annotations

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_pieces_of_the_corners(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.run(["/usr/bin/g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "celeris_b200", "csrc"),
                    os.path.join(ROOT, "tests", "corner_pieces_check.cpp"), "-o", exe], check=True)
    corners, uncovered, too_large, wrong = map(int, subprocess.run([exe], capture_output=True, text=True,
                                                                   check=True).stdout.split())
    assert corners > 10000
    assert uncovered == 0 and wrong == 0
    assert too_large == 0
