"""The wide nodes' child codes name the children their meta bytes describe: compiles
tests/node_codes_check.cpp against the host builder and runs it (trees of 1 to 20000
primitives: a leaf-only root, a full root, ragged last levels)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "goodphotons_b200", "csrc")


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_child_codes_match_meta_bytes(tmp_path):
    exe = str(tmp_path / "node_codes_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, os.path.join(ROOT, "tests", "node_codes_check.cpp"),
                    os.path.join(CSRC, "bvh_build.cpp"), "-o", exe], check=True, capture_output=True, text=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    lines = r.stdout.strip().splitlines()
    assert r.returncode == 0, r.stdout + r.stderr
    assert len(lines) == 9 and all(l.endswith(": ok") for l in lines), r.stdout
