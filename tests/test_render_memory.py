"""The host side of renders -- device memory that runs out, launches that fail, the order of rays
that a tuning asks for: compiles and runs
tests/render_memory_check.cpp, in which goodphotons_b200/csrc/ftb_api.cpp runs on a CUDA
runtime made of host memory."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "goodphotons_b200", "csrc")
CUDA = next((d for d in (os.environ.get("CUDA_HOME", ""), "/usr/local/cuda")
             if os.path.exists(os.path.join(d, "include", "cuda_runtime.h"))), None)


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if shutil.which("g++") is None or CUDA is None:
        pytest.skip("needs g++ and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("render_memory") / "check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-I", os.path.join(CUDA, "include"), "-I", CSRC,
                    os.path.join(ROOT, "tests", "render_memory_check.cpp"), os.path.join(CSRC, "bvh_build.cpp"),
                    "-o", exe], check=True, capture_output=True, text=True)

    def run(what):
        r = subprocess.run([exe, what], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0 and r.stdout.strip().endswith(f"{what}: ok"), r.stdout + r.stderr
    return run


def test_no_error_is_left_on_the_thread(check):
    check("error_left_behind")


def test_nothing_is_in_flight_after_a_failed_render(check):
    check("second_buffer")


def test_buffers_stay_within_the_stated_footprint(check):
    check("stated_memory")


def test_rays_are_ordered_as_the_tuning_says(check):
    check("ray_order")
