"""Tables, flags and constants reach the device before any stream's kernel can read
them: no source file uploads or clears device memory on the default stream, which
non-blocking streams do not wait for (cudaMemcpy from pageable memory may return
before its transfer has ended, cudaMemset does). upload_table / fill_table wait."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "stream-k-gemm_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh", ".h")))
DEFAULT_STREAM = re.compile(
    r"cudaMemset\s*\(|cudaMemcpyToSymbol\s*\(|cudaMemcpy\s*\([^;]*cudaMemcpyHostToDevice[^;]*;",
    re.S)


@pytest.mark.parametrize("name", SOURCES)
def test_no_upload_on_the_default_stream(name):
    with open(os.path.join(CSRC, name)) as f:
        code = re.sub(r"//[^\n]*", "", f.read())
    found = [m.group(0).split("\n")[0] for m in DEFAULT_STREAM.finditer(code)]
    assert not found, found
