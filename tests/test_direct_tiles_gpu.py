"""The plain method's tiled kernel: explicit tiles, rows too wide for the cyclic
form, and its split of a tile's rows, against the oracle.  (The default form of
ordinary sizes is the cyclic kernel.)  Widths of a multiple of 16 bytes take the
TMA loader, others cp.async.

Bounds: the FP32 gate 1e-5 of max|oracle| and 1e-12 for FP64, as the other
tests of the plain method."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT
from helpers import rel_to_max, seeded
from oracle import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import xcorr  # noqa: E402

TOL = {"f32": 1e-5, "f64": 1e-12}
# around the tiles' edges (32 and 64 shifts), 128-column chunks, 8 and 4 partners
SHAPES = [
    ("one_to_one", 1, 1, (1, 1), (1, 1)), ("one_to_one", 1, 1, (33, 65), (33, 65)),
    ("one_to_one", 1, 1, (32, 64), (33, 64)), ("one_to_one", 1, 1, (130, 131), (7, 200)),
    ("one_to_many", 1, 9, (64, 64), (64, 64)), ("one_to_many", 1, 5, (37, 150), (61, 3)),
    ("n_to_mn", 3, 9, (29, 29), (29, 29)), ("n_to_m", 2, 5, (48, 20), (16, 52)), ("n_to_m", 3, 3, (70, 1), (5, 1)),
    # more tiles than a wave of CTAs: rows are not split
    ("one_to_many", 1, 90, (70, 140), (20, 132)),
]


def run(mode, left, right, method):
    out = torch.full((xcorr.output_count(mode, len(left), len(right)), left.shape[1] + right.shape[1] - 1,
                      left.shape[2] + right.shape[2] - 1), float("nan"),
                     dtype=torch.float32 if left.dtype == np.float32 else torch.float64, device="cuda")
    xcorr.correlate(mode, torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda(), method=method, out=out)
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("tile", [1, 2, 3])
@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("shape", SHAPES, ids=[f"{s[0]}-{s[3]}-{s[4]}" for s in SHAPES])
def test_explicit_tiles(shape, dtype, tile):
    mode, n, m, ls, rs = shape
    npdt = np.float32 if dtype == "f32" else np.float64
    left, right = seeded((n,) + ls, 41, "signed", npdt), seeded((m,) + rs, 42, "signed", npdt)
    ref = oracle.run_mode(mode, left, right, dtype="f32acc64" if dtype == "f32" else "f64", threads=8)
    assert rel_to_max(run(mode, left, right, f"direct:{tile}"), ref) <= TOL[dtype]


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("wl,wr", [(64, 32), (64, 36), (62, 32), (61, 35)])
def test_loaders(wl, wr, dtype):
    """Both sides aligned, the right's rows, the left's rows and neither a
    multiple of 16 bytes."""
    npdt = np.float32 if dtype == "f32" else np.float64
    left, right = seeded((2, 40, wl), 7, "normal", npdt), seeded((4, 24, wr), 8, "normal", npdt)
    ref = oracle.run_mode("n_to_mn", left, right, dtype="f32acc64" if dtype == "f32" else "f64", threads=8)
    for tile in (1, 2, 3):
        assert rel_to_max(run("n_to_mn", left, right, f"direct:{tile}"), ref) <= TOL[dtype]


@pytest.mark.parametrize("suffix", ["f32", "f64"])
def test_split_rows_add_into_the_callers_output(suffix):
    """Rows beyond the cyclic form's reach through a launcher that adds: the
    output starts at 1 and ends at 1 plus the correlation."""
    npdt, dt = (np.float32, torch.float32) if suffix == "f32" else (np.float64, torch.float64)
    rows, cols = (12, 2100) if suffix == "f32" else (12, 16500)
    left, right = seeded((1, rows, cols), 43, "signed", npdt), seeded((1, rows, cols), 44, "signed", npdt)
    out = torch.full((1, 2 * rows - 1, 2 * cols - 1), 1.0, dtype=dt, device="cuda")
    dl, dr = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    fn = getattr(xcorr.lib(), f"xc_run_ccn_shuffle_work_distribution_{suffix}")
    xcorr.check(fn(dl.data_ptr(), dr.data_ptr(), out.data_ptr(), xcorr.size2(rows, cols),
                   xcorr.size2(2 * rows - 1, 2 * cols - 1), 8, 4, 1, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    ref = oracle.run_mode("one_to_one", left, right, dtype="f32acc64" if suffix == "f32" else "f64", threads=8)
    assert rel_to_max(out.cpu().numpy().astype(np.float64) - 1.0, ref) <= TOL[suffix]


SLICED = """
import sys
sys.path[:0] = [{tests!r}, {root!r}, {pkg!r}]
import numpy as np, torch, xcorr
from helpers import rel_to_max, seeded
from oracle import oracle
left, right = seeded((2, 50, 70), 45, "signed"), seeded((8, 41, 33), 46, "signed")
ref = oracle.run_mode("n_to_m", left, right, dtype="f32acc64", threads=8)
for tile in (1, 2, 3):
    out = xcorr.correlate("n_to_m", torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda(), method=f"direct:{{tile}}")
    torch.cuda.synchronize()
    assert rel_to_max(out.cpu().numpy(), ref) <= 1e-5, tile
"""


@pytest.mark.parametrize("rows", [1, 5, 41, 1000])
def test_fixed_slices(rows):
    """XC_DIRECT_SLICE_ROWS (read once per process): one row, a remainder, all
    rows and more."""
    code = SLICED.format(tests=os.path.join(ROOT, "tests"), root=ROOT, pkg=os.path.join(ROOT, "cross-corr_gb300"))
    subprocess.run([sys.executable, "-c", code], check=True, env=dict(os.environ, XC_DIRECT_SLICE_ROWS=str(rows)),
                   timeout=240)
