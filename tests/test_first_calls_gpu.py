"""The first call for a shape and a plan's first execution on a non-blocking
stream, right after the plan's tables were made: the same bits as a repeated
call.  (These kernels add nothing atomically, so a repeat is exact.)"""
import numpy as np
import pytest

from helpers import seeded

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import xcorr  # noqa: E402


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("mode,n,m,side", [("one_to_one", 1, 1, 23), ("one_to_many", 1, 70, 67),
                                           ("n_to_m", 5, 40, 61), ("one_to_many", 1, 3, 1211)])
def test_first_fft_call_on_a_side_stream(mode, n, m, side, dtype):
    npdt = np.float32 if dtype == "f32" else np.float64
    left = torch.from_numpy(seeded((n, side, side), 81, "signed", npdt)).cuda()
    right = torch.from_numpy(seeded((m, side, side + 1), 82, "signed", npdt)).cuda()
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        first = xcorr.correlate(mode, left, right, method="fft")
        again = xcorr.correlate(mode, left, right, method="fft")
    torch.cuda.synchronize()
    assert torch.isfinite(first).all() and torch.equal(first, again)


def test_first_ragged_execution_on_a_side_stream():
    rng = np.random.default_rng(83)
    sides = rng.integers(150, 420, (12, 4)).tolist()
    lefts = [rng.uniform(-1, 1, (a, b)).astype(np.float32) for a, b, _, _ in sides]
    rights = [rng.uniform(-1, 1, (c, d)).astype(np.float32) for _, _, c, d in sides]
    plan = xcorr.RaggedPlan(lefts, rights, [(k, k) for k in range(len(sides))])
    torch.cuda.synchronize()  # the inputs are there; the variant's tables are made next
    plan.select(plan.describe()["n_variants"] - 2)  # every pair on the FFT kernels
    assert plan.describe()["tc_pairs"] == len(sides)
    with torch.cuda.stream(torch.cuda.Stream()):
        plan.execute()
        first = plan.out.clone()
        plan.execute()
        again = plan.out.clone()
    torch.cuda.synchronize()
    assert torch.isfinite(first).all() and torch.equal(first, again)
    plan.close()
