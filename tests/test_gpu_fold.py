"""The ordered history fold (csrc/mc_fold.cuh) gives the serial chain's bits
(tests/fold_check.cu), and a replay long enough for several of its steps
equals the oracle."""
import os
import subprocess

import numpy as np
import pytest

from helpers import same_bits

ROOT = os.path.abspath(os.path.join(os.path.dirname(__file__), ".."))
pytestmark = pytest.mark.gpu


def test_fold_equals_the_serial_chain(tmp_path):
    exe = str(tmp_path / "fold_check")
    nvcc = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", "-fmad=false",
                        "-Xcompiler", "-ffp-contract=off", "-I", os.path.join(ROOT, "mc-old_gb300", "csrc"),
                        os.path.join(ROOT, "tests", "fold_check.cu"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


@pytest.mark.parametrize("n", [4096, 20011])
def test_long_replay_equals_the_oracle(oracle_lib, tmp_path, n):
    import mcgpu
    from mcgpu import workloads as W
    d = W.mg_layered_slab(str(tmp_path), n_regions=4, detectors=True)
    p = mcgpu.Problem(d)
    p.run(n=n, seed=7, mode="replay")
    _, _, s, q = p.all_tallies()
    p.close()
    r = oracle_lib.run(oracle_lib.load(d), n=n, seed=7)
    assert np.count_nonzero(r.sum) >= 4
    assert same_bits(s, r.sum) and same_bits(q, r.sq)
