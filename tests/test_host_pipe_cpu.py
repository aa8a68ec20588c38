"""The chunked host-pointer calls when a chunk's launch fails: the threads that upload
stop before the call's final wait, so no copy still reads the pinned slots or writes the
staging buffers when the next call starts. Run on a stand-in for the CUDA runtime."""
import os
import subprocess

import pytest

import skgemm

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(REPO, "tests", "cpp", "host_pipe.cpp")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("pipe") / "host_pipe")
    cxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else "g++"
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(REPO, "include"),
                    "-I", os.path.join(REPO, "stream-k-gemm_b200", "csrc"),
                    "-I", os.path.join(CUDA, "include"), SRC, "-o", out, "-lpthread", "-ldl"],
                   check=True, capture_output=True, text=True)
    return out


@pytest.mark.parametrize("mode", ["fail", "ok", "unpinned", "pinned"])
def test_no_copy_outlives_the_call(exe, mode):
    r = subprocess.run([exe, mode], capture_output=True, text=True, timeout=60, check=True)
    st, seen, late, after, whole, left = map(int, r.stdout.split())
    assert late == 0 and after == 0
    assert left == 0  # slots that cannot be pinned: the driver copies, nothing else changes
    if mode != "fail":  # pinned, unpinned: the driver copies, one chunk ahead of its event
        assert st == skgemm.OK and whole == 1 and seen >= 8
    else:
        assert st == skgemm.ERR_OOM and 0 < seen < 32
