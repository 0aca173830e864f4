"""Work lists of the list engine: every position in exactly one short segment,
medium segment or piece (tests/cpp/segbook_test.cpp)."""
from __future__ import annotations

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_segment_lists_cover_every_position(tmp_path):
    exe = tmp_path / "segbook_test"
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", str(exe),
                    os.path.join(ROOT, "tests", "cpp", "segbook_test.cpp")], check=True)
    assert subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.strip() == "ok"
