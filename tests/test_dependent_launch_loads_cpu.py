"""The preparation kernels of the split tensor-core path start under the kernel
before them and wait for it (griddepcontrol.wait) before they read what it
wrote.  The compiler may move a non-coherent load above that wait, so what an
earlier kernel wrote is read neither by __ldg nor through __restrict__ pointers,
and the sums that the previous launch adds up atomically only by ld_after.
Which loads the compiler moves is its own choice, so the source is checked."""
import os
import re

from conftest import ROOT

SOURCE = os.path.join(ROOT, "cross-corr_gb300", "csrc", "tc_bf16x3.cu")


CHAIN = ["sum_block", "mean_sd", "window_block", "split_block", "colsum_block", "colsum_kernel", "rowscan_kernel"]


def test_no_movable_loads_behind_the_wait():
    text = re.sub(r"//[^\n]*", "", open(SOURCE).read())
    for name in CHAIN:
        body = re.search(r"^__(?:device|global)__[^;{]*\b%s\(.*?\n}\n" % name, text, re.S | re.M).group(0)
        assert "__ldg(" not in body, name
        assert "__restrict__" not in body, name
        reads = re.findall(r"(?<![&\w.])(?:sd_\.|wa\.)?(?:sums|sq)\[", body)
        assert not reads, (name, reads)
