"""The mixed engine's test that a flight ends before a sphere for certain, for
directions of any length (tests/sphere_direction_check.cu, built with the
engine's arithmetic flags)."""
import os
import subprocess

import pytest

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
pytestmark = pytest.mark.gpu


def test_any_length_of_direction(tmp_path):
    exe = str(tmp_path / "sphere_direction_check")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-ftz=true",
                        "-prec-div=false", "-prec-sqrt=false", "-I", os.path.join(ROOT, "mc-old_gb300", "csrc"),
                        "-I", os.path.join(ROOT, "include"), os.path.join(ROOT, "tests", "sphere_direction_check.cu"), "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
