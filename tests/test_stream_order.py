"""Sessions run their kernels on streams that do not wait for the default
stream, and a copy from pageable memory on the default stream may return before
the device has the data: what such a stream's kernels read is copied on that
stream."""
import glob
import os
import re

import hydrofv_gb300 as H

GPU = os.path.join(H.PKG, "csrc", "gpu")


def units():
    for path in sorted(glob.glob(os.path.join(GPU, "*.cu"))):
        text = re.sub(r'"[^"\n]*"', '""', open(path).read())      # (messages name the calls)
        if "cudaStreamNonBlocking" in text:
            yield os.path.basename(path), text


def test_there_are_such_units():
    assert {"runtime2d.cu", "runtime_batch.cu", "adjoint2d.cu"} <= {name for name, _ in units()}


def test_uploads_are_on_the_session_s_stream():
    bad = [(name, call) for name, text in units()
           for call in re.findall(r"\bcudaMem(?:cpy|cpy2D|set)\([^;]*;", text)
           if not re.search(r"\bcudaMemcpyDeviceToHost\b", call)]
    assert bad == []
