"""Rules of the whole-state reads that need no GPU, over a runtime of host memory (readback_check.cpp)."""
from __future__ import annotations

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("readback") / "check")
    subprocess.run(["/usr/bin/g++", "-O2", "-std=c++17", "-I", "/usr/local/cuda/include", "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(ROOT, "celeris_b200", "csrc"), os.path.join(ROOT, "tests", "readback_check.cpp"),
                    os.path.join(ROOT, "celeris_b200", "csrc", "readback.cpp"), "-o", exe, "-lpthread"], check=True)
    return lambda rule: subprocess.run([exe, rule], capture_output=True, text=True, check=True, timeout=120).stdout.strip()


@pytest.mark.parametrize("rule", ["slots", "refused", "device", "pinned", "thread"])
def test_read_rule(check, rule):
    assert check(rule) == "ok"
