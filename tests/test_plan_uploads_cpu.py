"""Tables that plans copy to the device are there before any stream's kernels
can read them.  A host-to-device cudaMemcpy from pageable memory may return
before the copy has reached the device and orders only the legacy default
stream after it, so every such copy goes through upload(), which waits.  The
order cannot be provoked, so the sources are checked."""
import glob
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "cross-corr_gb300", "csrc")


def code(path):
    return re.sub(r"//[^\n]*", "", open(path).read())


def test_only_upload_copies_synchronously_and_it_waits():
    copies = {}
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        n = len(re.findall(r"\bcudaMemcpy(?:2D|3D|ToSymbol)?\s*\(", code(path)))
        if n:
            copies[os.path.basename(path)] = n
    assert copies == {"xc_runtime.cu": 1}
    body = re.search(r"xc_status upload\(.*?\n}\n", code(os.path.join(CSRC, "xc_runtime.cu")), re.S).group(0)
    copy, wait = body.find("cudaMemcpy("), body.find("cudaStreamSynchronize(cudaStreamLegacy)")
    assert 0 < copy < wait
