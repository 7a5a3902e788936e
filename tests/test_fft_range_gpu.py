"""Small FP32 inputs through the fused FFT kernels of uniform problems: scaled
by a power of two they give the scaled result, although the spectra and their
products come near the smallest normal number, on either side alone and on both,
in every form of the pipeline (both transforms in the column kernel, left
spectra made first, all spectra made first).  Large inputs do as far as the
separate transforms, scaled at the end, do, and beyond.

Bound: the two runs differ by what the scaled one rounds below 2^-126.  Results
here are 2^-124 and more, whose last place is 2^-147; the bound of two runs of
the same transforms elsewhere, 1e-6 of max|out|, is 14 of them or more."""
import numpy as np
import pytest

from helpers import rel_to_max, seeded

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import xcorr  # noqa: E402


@pytest.mark.parametrize("el,er", [(-126, 0), (0, -126), (-66, -66), (50, 50)])
@pytest.mark.parametrize("mode,n,m,ls,rs", [("one_to_one", 1, 1, (256, 256), (256, 256)),
                                            ("one_to_many", 1, 24, (256, 256), (240, 256)),
                                            ("n_to_m", 4, 20, (200, 230), (256, 220)),
                                            ("one_to_many", 1, 2, (1100, 1100), (1100, 1100))])
def test_scaled_inputs_give_the_scaled_result(mode, n, m, ls, rs, el, er):
    left, right = seeded((n,) + ls, 61, "normal"), seeded((m,) + rs, 62, "normal")
    got = []
    for a, b in ((0, 0), (el, er)):
        out = xcorr.correlate(mode, torch.from_numpy(np.ldexp(left, a)).cuda(),
                              torch.from_numpy(np.ldexp(right, b)).cuda(), method="fft")
        got.append(np.ldexp(out.cpu().numpy().astype(np.float64), -a - b))
    assert np.isfinite(got[1]).all()
    assert rel_to_max(got[1], got[0]) <= 1e-6
