"""The library works on streams that do not wait for the default one, and a
default-stream copy from pageable memory may return before it has arrived.  So
no source uploads or clears device memory there: each does on the stream of the
kernels that follow."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "calypso_b200", "csrc")


def test_no_uploads_on_the_default_stream():
    files = sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh")))
    assert files
    for f in files:
        text = open(f).read()
        for call in re.findall(r"\bcudaMemcpy\s*\([^;]*;", text):
            assert "cudaMemcpyDeviceToHost" in call, (os.path.basename(f), call)
        assert not re.search(r"\bcudaMemset\s*\(", text), os.path.basename(f)
