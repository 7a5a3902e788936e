"""The part of the Toeplitz buffer that the split tensor-core kernel's builder
warps write covers every operand its MMAs read (tc_core_check.cpp, compiled
from the header the kernel uses), over widths around every rounding edge."""
import os
import subprocess

from conftest import ROOT

CSRC = os.path.join(ROOT, "cross-corr_gb300", "csrc")
HERE = os.path.dirname(os.path.abspath(__file__))
WIDTHS = [1, 2, 7, 8, 15, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 200, 240, 255, 256, 257, 300, 511, 512, 513,
          700, 1024, 2048]


def test_core_matrices_cover_every_window(tmp_path):
    exe = str(tmp_path / "tc_core_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", CSRC, os.path.join(HERE, "tc_core_check.cpp"), "-o", exe],
                   check=True)
    cases = [(wl, wr, tf) for wl in WIDTHS for wr in WIDTHS for tf in (0, 1)]
    out = subprocess.run([exe], input="\n".join("%d %d %d" % c for c in cases), capture_output=True, text=True,
                         check=True).stdout.strip().splitlines()
    assert len(out) == len(cases)
    for c, line in zip(cases, out):
        assert line.startswith("ok"), (c, line)
