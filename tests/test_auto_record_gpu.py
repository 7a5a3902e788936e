"""XC_METHOD_AUTO without a network runs the algorithm that the exhaustive
autotune measured, returned and remembered for the problem, tile included.

Which kernel ran is told by a non-finite input: the tiled forms of the plain
kernel make NaN of an infinity in shifts that do not meet it (their tiles are
padded with zeros), the default form does not."""
import numpy as np
import pytest

from helpers import seeded

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import xcorr  # noqa: E402
from xcorr import selector  # noqa: E402


@pytest.mark.parametrize("side", [5, 8])
def test_auto_runs_the_remembered_tile(side):
    # one small FP64 pair: the split paths do not take it, and a transform is many launches
    left = torch.from_numpy(seeded((1, side, side), 91, dtype=np.float64)).cuda()
    right = torch.from_numpy(seeded((1, side - 1, side), 92, dtype=np.float64)).cuda()
    out = xcorr.correlate("one_to_one", left, right)
    selector.install(None)
    try:
        best, ms = selector.autotune("one_to_one", left, right, out)
        assert best.startswith("direct:") and ms > 0
        assert selector.select("one_to_one", "f64", (side, side), 1, (side - 1, side), 1) == best
        masks = {m: [] for m in ("auto", best, "direct")}
        for x in range(side):  # one infinity in the right's first row, column after column
            met = right.clone()
            met[0, 0, x] = float("inf")
            for m in masks:
                masks[m].append(torch.isnan(xcorr.correlate("one_to_one", left, met, method=m)))
    finally:
        selector.install("builtin")
    masks = {m: torch.stack(v) for m, v in masks.items()}
    assert not torch.equal(masks[best], masks["direct"])
    assert torch.equal(masks["auto"], masks[best])
