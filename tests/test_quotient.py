"""The sweeps' quotient by a prepared mass (velox_b200/csrc/quotient.cuh) is the
IEEE quotient over the ranges that it claims, on the host (same operations)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_quotient_equals_division(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ is missing")
    out = str(tmp_path / "quotient_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-mfma", "-ffp-contract=off", "-I",
                    os.path.join(ROOT, "velox_b200", "csrc"), os.path.join(ROOT, "tests", "quotient_check.cpp"),
                    "-o", out], check=True)
    assert subprocess.run([out], capture_output=True, text=True).stdout.strip() == "0"
