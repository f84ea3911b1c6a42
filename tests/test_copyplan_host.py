"""Copy-block plans on the host (tests/cpp/copyplan_test.cpp), under AddressSanitizer and
UndefinedBehaviorSanitizer: lists replanned for the other down-tile edge, and the RGB8 canvas plane."""
from __future__ import annotations

import subprocess
from pathlib import Path

from test_host_abi import _sanitized_build

REPO = Path(__file__).resolve().parents[1]


def test_replanned_lists_and_rgb_canvas_plane(tmp_path):
    csrc = REPO / "hm-cupano_gb300" / "csrc"
    exe = _sanitized_build(tmp_path, "copyplan", [REPO / "tests" / "cpp" / "copyplan_test.cpp", csrc / "hmp_plan.cpp",
                                                  csrc / "hmp_copyplan.cpp"], "g++")
    r = subprocess.run([str(exe), "400", "3"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr[-2000:]
    planned, planes = (int(v) for v in r.stdout.split()[1::2])
    assert planned > 100 and planes > 100
