"""The serving scheduler reads the device error word of each request (or grouped
launch) when it completes: a failed one ends the run there with the request's index
and shape, instead of counting as completed until the last request. The scheduler
runs here on an executor that stands in for the device."""
import os
import shutil
import subprocess

import pytest

import skgemm

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(REPO, "tests", "cpp", "serve_errors.cu")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
pytestmark = pytest.mark.skipif(not (os.path.exists(NVCC) or shutil.which(NVCC)),
                                reason="needs nvcc")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("serve") / "serve_errors")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    "-I", os.path.join(REPO, "include"),
                    "-I", os.path.join(REPO, "stream-k-gemm_b200", "csrc"), SRC, "-o", out],
                   check=True, capture_output=True, text=True)
    return out


def run(exe, kind, bad):
    r = subprocess.run([exe, kind, str(bad)], capture_output=True, text=True, timeout=60, check=True)
    st, ran, msg = r.stdout.split(" ", 2)
    return int(st), int(ran), msg, r.stderr


@pytest.mark.parametrize("kind", ["native", "ozaki"])
def test_failed_request_ends_the_run_at_its_completion(exe, kind):
    assert run(exe, kind, -1)[:2] == (skgemm.OK, 6)
    st, ran, msg, err = run(exe, kind, 2)
    assert st == skgemm.ERR_DEVICE_TIMEOUT and ran == 2
    assert "request 2 (Ng 1632, nb 32)" in msg and "word" in msg
    assert "request 2 (Ng 1632, nb 32)" in err  # said before the teardown waits
