"""The bake's parallel loops cover every index once: compiles and runs
tests/parallel_for_check.cpp against goodphotons_b200/csrc/bvh_build.h."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_every_index_once(tmp_path):
    exe = str(tmp_path / "parallel_for_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "goodphotons_b200", "csrc"),
                    os.path.join(ROOT, "tests", "parallel_for_check.cpp"), "-o", exe],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    lines = r.stdout.strip().splitlines()
    assert r.returncode == 0 and len(lines) == 11 and all(l.endswith(": ok") for l in lines), r.stdout
