"""The plain method's kernel by cyclic column classes against the oracle, where
its dispatch can go wrong: classes and right blocks that do not fill their 32
bytes, lefts narrower than the rights (several wraps per lane), single rows
and columns, row blocks with a remainder, the windowed form of wide lefts
(with and without a wrap inside the window), rows too wide for it, and the
launchers that add into the caller's output.

Bounds: the FP32 gate 1e-5 of max|oracle| and 1e-12 for FP64, as the other
tests of the plain method.
"""
import numpy as np
import pytest

from helpers import rel_to_max, seeded
from oracle import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import xcorr  # noqa: E402

TOL = {"f32": 1e-5, "f64": 1e-12}
SHAPES = [
    ((1, 1), (1, 1)), ((1, 9), (1, 7)), ((9, 1), (7, 1)), ((5, 3), (4, 100)), ((3, 1), (2, 33)),
    ((8, 8), (8, 8)), ((17, 31), (16, 33)), ((40, 32), (33, 32)), ((33, 250), (19, 8)), ((30, 23), (75, 59)),
    ((12, 513), (9, 15)), ((10, 700), (18, 640)), ((6, 1030), (35, 16)), ((64, 64), (64, 64)),
]


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("ls,rs", SHAPES, ids=[f"{a}-{b}" for a, b in SHAPES])
@pytest.mark.parametrize("mode,n,m", [("one_to_one", 1, 1), ("n_to_mn", 2, 4), ("n_to_m", 3, 2)])
def test_shapes(mode, n, m, ls, rs, dtype):
    npdt = np.float32 if dtype == "f32" else np.float64
    left, right = seeded((n,) + ls, 31, "signed", npdt), seeded((m,) + rs, 32, "signed", npdt)
    ref = oracle.run_mode(mode, left, right, dtype="f32acc64" if dtype == "f32" else "f64", threads=8)
    out = torch.full(ref.shape, float("nan"), dtype=torch.float32 if dtype == "f32" else torch.float64, device="cuda")
    xcorr.correlate(mode, torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda(), out=out)
    torch.cuda.synchronize()
    assert rel_to_max(out.cpu().numpy(), ref) <= TOL[dtype]


def test_many_outputs_fill_the_longer_blocks():
    """Enough warps for every block length (16 rows and 8-warp CTAs at the
    largest), on unaligned rows."""
    for n, ls, rs in ((40, (70, 61), (50, 37)), (160, (70, 61), (50, 37)), (12, (90, 301), (33, 21))):
        left, right = seeded((1,) + ls, 33, "normal"), seeded((n,) + rs, 34, "normal")
        ref = oracle.run_mode("one_to_many", left, right, dtype="f32acc64", threads=8)
        out = xcorr.correlate("one_to_many", torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda())
        torch.cuda.synchronize()
        assert rel_to_max(out.cpu().numpy(), ref) <= TOL["f32"]


def test_rows_too_wide_keep_the_tiled_kernel():
    left, right = seeded((1, 3, 9000), 35, "signed"), seeded((1, 2, 5000), 36, "signed")
    ref = oracle.run_mode("one_to_one", left, right, dtype="f32acc64", threads=8)
    out = xcorr.correlate("one_to_one", torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda())
    torch.cuda.synchronize()
    assert rel_to_max(out.cpu().numpy(), ref) <= TOL["f32"]


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("ls,rs", [((32, 32), (32, 32)), ((17, 33), (9, 21)), ((5, 3), (7, 50)), ((64, 300), (64, 40)),
                                   ((6, 1030), (35, 16))])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_non_finite_values_stay_where_they_are_met(value, ls, rs, dtype):
    """One non-finite value reaches the shifts that multiply it and no others
    (the kernel's zero columns and rows would make NaN of it elsewhere): the
    others equal, within the method's bound, the result with a zero there."""
    npdt = np.float32 if dtype == "f32" else np.float64
    for side, at in [(s, (int(fy * (h - 1)), int(fx * (w - 1)))) for s, (h, w) in ((0, ls), (1, rs))
                     for fy, fx in ((0, 0), (1, 1), (1, 0), (0.5, 0.5))]:
        pair = [seeded((1,) + ls, 37, "uniform", npdt) + npdt(0.5), seeded((1,) + rs, 38, "uniform", npdt) + npdt(0.5)]
        pair[side][0][at] = 0
        ref = oracle.run_mode("one_to_one", *pair, dtype="f32acc64" if dtype == "f32" else "f64", threads=4)[0]
        mark = [np.zeros_like(pair[0]), np.ones_like(pair[1])] if side == 0 else [np.ones_like(pair[0]), np.zeros_like(pair[1])]
        mark[side][0][at] = 1
        met = oracle.run_mode("one_to_one", *mark, dtype="f32acc64" if dtype == "f32" else "f64", threads=4)[0] > 0.5
        pair[side][0][at] = value
        out = xcorr.correlate("one_to_one", *[torch.from_numpy(x).cuda() for x in pair])[0].cpu().numpy()
        assert np.array_equal(~np.isfinite(out), met)
        assert np.array_equal(np.isnan(out), met if np.isnan(value) else np.zeros_like(met))
        assert rel_to_max(np.where(met, 0, out), np.where(met, 0, ref)) <= TOL[dtype]
