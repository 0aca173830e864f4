"""The largest plan of the list engine (tests/cpp/seglimit_test.cpp)."""
from __future__ import annotations

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_positions_stay_below_the_wrap(tmp_path):
    exe = tmp_path / "seglimit_test"
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", "seglimit_test.cpp")], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.strip() == "ok"
