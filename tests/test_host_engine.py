"""The host side of the engines over a fake CUDA runtime (tests/fake_cudart.cpp),
which keeps device memory on the host, runs no kernel and fails where it is
told to: tests/host_engine_check.cpp, linked with the library's own objects."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")


@pytest.fixture(scope="module")
def check(tmp_path_factory):
    if shutil.which("g++") is None or not os.path.isdir(CUDA_INC):
        pytest.skip("g++ or the CUDA headers are missing")
    import build as B
    B.build()
    from mcgpu import workloads as W
    d = tmp_path_factory.mktemp("host_engine")
    objs = [os.path.join(B.BUILD, name + ".o") for name, _ in B.SOURCES]
    exe = str(d / "check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-I", CUDA_INC, "-I", os.path.join(ROOT, "include"),
                        "-I", B.CSRC, os.path.join(ROOT, "tests", "host_engine_check.cpp"),
                        os.path.join(ROOT, "tests", "fake_cudart.cpp"), *objs, "-lpthread", "-o", exe],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    ce = W.ce_sphere(str(d / "ce"), n_points=300, n_spectrum=10)
    mg = W.mg_layered_slab(str(d / "mg"), n_regions=4, detectors=True)
    wide = W.mg_layered_slab(str(d / "wide"), n_regions=4)
    many = "".join(f'<estimator name="w{i}" scores="flux"><cell name="c{i % 4}"/><filter type="energy" grid_linear="0 1 {k}"/></estimator>'
                   for i, k in enumerate((10_000, 10_002)))     # with the transmitted current 20,003 bins
    with open(wide + "/input.xml") as f:
        s = f.read()
    with open(wide + "/input.xml", "w") as f:
        f.write(s.replace("</estimators>", many + "</estimators>"))

    def run(scenario):
        r = subprocess.run([exe, scenario, ce, os.path.join(ce, "xs_library"), mg, wide, str(d)], capture_output=True, text=True,
                           timeout=300)
        assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout[-3000:] + r.stderr[-1000:]
    return run


@pytest.mark.parametrize("scenario", ["concurrent reads", "not loaded", "deeper stack", "failed query", "failed reduce",
                                      "failed calls", "noalloc clears", "launch shape", "row bound",
                                      "state keys"])
def test_host_engine(check, scenario):
    check(scenario)
