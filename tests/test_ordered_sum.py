"""The stabiliser's mean flow is the reference's sum in feature order; the kernel forms it by scans of
whole units (hm-cupano_gb300/csrc/hmp_ordered_sum.h). The header's host build against the plain
sequential sum, bit for bit, on sums that drift, hover at zero, tie, and overflow."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]


def test_ordered_sum_equals_the_sequential_sum(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no g++")
    exe = tmp_path / "ordered_sum"
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(REPO / "hm-cupano_gb300" / "csrc"),
                    str(REPO / "tests" / "cpp" / "ordered_sum_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
