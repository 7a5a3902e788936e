"""The plain method's cyclic kernel on thin matrices against the oracle: rights
of one row (one row shift per lane, or two where a single column block fills the
GPU), and narrow lefts that keep their part although the right is wider (few
right rows, many left rows), whose lanes wrap more than once.

Bounds: the FP32 gate 1e-5 of max|oracle| and 1e-12 for FP64, as the other
tests of the plain method."""
import numpy as np
import pytest

from helpers import rel_to_max, seeded
from oracle import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import xcorr  # noqa: E402

TOL = {"f32": 1e-5, "f64": 1e-12}
CASES = [
    # one right row: single pairs, several column blocks, windowed lefts, one column block of a full launch
    ("one_to_one", 1, 1, (1, 1), (1, 1)), ("one_to_one", 1, 1, (1, 300), (1, 40)), ("one_to_one", 1, 1, (7, 33), (1, 33)),
    ("n_to_m", 2, 3, (5, 1900), (1, 17)), ("n_to_mn", 3, 6, (16, 300), (1, 301)), ("one_to_many", 1, 40, (150, 203), (1, 5)),
    # narrow lefts in their place: up to 8 right columns; and from 9000 (16000) lanes on, either side of the rule
    ("one_to_one", 1, 1, (40, 1), (1, 8)), ("one_to_one", 1, 1, (9, 3), (1, 4)), ("one_to_many", 1, 16, (600, 4), (1, 61)),
    ("one_to_many", 1, 14, (600, 4), (1, 61)), ("one_to_many", 1, 70, (250, 3), (3, 40)), ("n_to_m", 6, 20, (64, 30), (1, 50)),
    ("n_to_mn", 4, 240, (67, 9), (2, 23)), ("one_to_many", 1, 300, (63, 9), (2, 23)),
]
IDS = [f"{c[0]}-{c[1]}-{c[2]}-{c[3]}-{c[4]}" for c in CASES]


def run(mode, left, right):
    out = torch.full((xcorr.output_count(mode, len(left), len(right)), left.shape[1] + right.shape[1] - 1,
                      left.shape[2] + right.shape[2] - 1), float("nan"),
                     dtype=torch.float32 if left.dtype == np.float32 else torch.float64, device="cuda")
    xcorr.correlate(mode, torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda(), out=out)
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("mode,n,m,ls,rs", CASES, ids=IDS)
def test_thin_shapes(mode, n, m, ls, rs, dtype):
    npdt = np.float32 if dtype == "f32" else np.float64
    left, right = seeded((n,) + ls, 51, "signed", npdt), seeded((m,) + rs, 52, "signed", npdt)
    ref = oracle.run_mode(mode, left, right, dtype="f32acc64" if dtype == "f32" else "f64", threads=8)
    assert rel_to_max(run(mode, left, right), ref) <= TOL[dtype]


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("n,m,ls,rs", [(1, 1, (40, 1), (1, 8)), (1, 16, (600, 4), (1, 61)), (1, 1, (3, 90), (1, 31))])
def test_an_infinity_reaches_the_shifts_that_meet_it(n, m, ls, rs, dtype):
    npdt = np.float32 if dtype == "f32" else np.float64
    left, right = seeded((n,) + ls, 53, "uniform", npdt) + npdt(0.5), seeded((m,) + rs, 54, "uniform", npdt) + npdt(0.5)
    for at in ((0, 0, 0), (0, ls[0] // 2, ls[1] - 1)):
        mark = np.zeros_like(left)
        mark[at] = 1
        met = oracle.run_mode("one_to_many", mark, np.ones_like(right), dtype="f64" if dtype == "f64" else "f32acc64",
                              threads=8) > 0.5
        bad = left.copy()
        bad[at] = np.inf
        assert np.array_equal(np.isinf(run("one_to_many", bad, right)), met)
        assert not np.isnan(run("one_to_many", bad, right)).any()
