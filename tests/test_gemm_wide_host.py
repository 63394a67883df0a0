"""How the GEMM for bf16 weights divides its work and its scratch (csrc/pi_gemm_wide.cuh): plain integer code, run here without a
GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lines(tmp_path_factory):
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    if not gxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path_factory.mktemp("cut") / "gemm_wide_cut")
    subprocess.run([gxx, "-std=c++17", "-O1", "-Wall", "-Wextra", "-Werror", os.path.join(ROOT, "tests", "cpp", "gemm_wide_cut.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    print(r.stdout)
    return r.stdout.split("\n")


@pytest.mark.parametrize("name", ["cut", "portions", "giving up", "dispatch"])
def test_plan(lines, name):
    assert f"ok {name}" in lines and not any(l.startswith("FAILED") for l in lines)
