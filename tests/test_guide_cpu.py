"""The host build's sampling guide tables (scene_build.cpp) against their definition."""
from __future__ import annotations

import os
import subprocess

from wobtoolbox_gb300 import build as B

HERE = os.path.dirname(os.path.abspath(__file__))


def test_guide_tables_are_their_definition(tmp_path):
    exe = tmp_path / "guide_check"
    subprocess.run([os.environ.get("CXX", "g++"), "-O2", "-std=c++17", "-ffp-contract=off", "-Wall", "-I", B.CSRC,
                    os.path.join(HERE, "guide_check.cpp"), os.path.join(B.CSRC, "scene_build.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "0 bad" in r.stdout, r.stdout[-2000:]
