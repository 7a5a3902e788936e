"""Every form of the fused FFT pipeline, at every transform length, against the
library transforms run stage by stage.  Sizes are chosen by the dispatch rule
(small FP64 problems keep the library transforms, short FP32 launches make no
spectra first), and each case checks by the plan's description that it runs the
form it is meant for, so that a change of the rule shows here.

Bounds: the error of either evaluation is at most its passes' roundings, about
log2 N (24) times a few units in the last place of max|out|: 1e-6 and 1e-14
each, as measured elsewhere below 5e-7 and 1e-15; twice the first, and ten times
the second for the differences.
"""
import numpy as np
import pytest

from helpers import seeded

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import xcorr  # noqa: E402

LENGTHS = [16, 32, 48, 64, 80, 96, 112, 128, 160, 192, 224, 256, 320, 384, 448, 512, 640, 768, 896, 1024, 1280, 1536,
           1792, 2048, 2560, 3072, 3584, 4096]
TOL = {"f32": 2e-6, "f64": 1e-13}


def describe(mode, dtype, ls, n, rs, m):
    plan = xcorr.FftPlan(mode, dtype, ls, n, rs, m)
    form = plan.describe()
    plan.close()
    return form


def check(mode, n, m, ls, rs, dtype):
    """Compares the fused result with the stages' and returns the form."""
    npdt = np.float32 if dtype == "f32" else np.float64
    left = torch.from_numpy(seeded((n,) + ls, 71, "signed", npdt)).cuda()
    right = torch.from_numpy(seeded((m,) + rs, 72, "signed", npdt)).cuda()
    plan = xcorr.FftPlan(mode, dtype, ls, n, rs, m)
    form = plan.describe()
    assert form["fused"] == 1
    ws = torch.empty(plan.workspace_bytes, dtype=torch.uint8, device="cuda")
    shape = (xcorr.output_count(mode, n, m), ls[0] + rs[0] - 1, ls[1] + rs[1] - 1)
    out = torch.full(shape, float("nan"), dtype=left.dtype, device="cuda")
    plan.execute(left, right, out, ws)
    ref = torch.empty(shape, dtype=left.dtype, device="cuda")
    s, L = torch.cuda.current_stream().cuda_stream, xcorr.lib()
    xcorr.check(L.xc_fft_forward(plan.handle, left.data_ptr(), right.data_ptr(), ws.data_ptr(), ws.numel(), s))
    xcorr.check(L.xc_fft_multiply(plan.handle, ws.data_ptr(), ws.numel(), s))
    xcorr.check(L.xc_fft_inverse(plan.handle, ref.data_ptr(), 1, ws.data_ptr(), ws.numel(), s))
    torch.cuda.synchronize()
    plan.close()
    err = (out - ref).abs().amax(dim=(1, 2)) / ref.abs().amax(dim=(1, 2))
    assert float(err.max()) <= TOL[dtype]  # (a NaN fails: nothing was left unwritten)
    return form


def thin(length, rows):
    """Shapes whose output is `length` by 16."""
    ls, rs = (13, length - 3), (4, 4)
    return (ls, rs) if not rows else (ls[::-1], rs[::-1])


@pytest.mark.parametrize("columns", [False, True])
@pytest.mark.parametrize("length", LENGTHS)
def test_fp64_lengths(length, columns):
    """Above 1.1 million points of output the FP64 kernels run with the left
    spectra first, above 2 million (n_to_m) with both sides'."""
    ls, rs = thin(length, columns)
    size = (length, 16) if columns else (16, length)
    form = check("one_to_many", 1, 1200 * 1024 // (16 * length) + 1, ls, rs, "f64")
    assert (form["size_y"], form["size_x"]) == size and form["spectra"] == 1
    form = check("n_to_m", 3, 2200 * 1024 // (3 * 16 * length) + 1, ls, rs, "f64")
    assert (form["size_y"], form["size_x"]) == size and form["spectra"] == 2


@pytest.mark.parametrize("columns", [False, True])
@pytest.mark.parametrize("length", LENGTHS)
def test_fp32_lengths(length, columns):
    """Short launches transform both sides' columns in the product kernel;
    with enough partners for more than a wave the spectra are made first."""
    ls, rs = thin(length, columns)
    size = (length, 16) if columns else (16, length)
    for mode, n, spectra in (("one_to_many", 1, 1), ("n_to_m", 2, 2)):
        m = 4
        while describe(mode, "f32", ls, n, rs, m)["spectra"] != spectra:
            m *= 2
            assert m <= 1 << 14
        form = check(mode, n, m + 1, ls, rs, "f32")
        assert (form["size_y"], form["size_x"], form["spectra"]) == size + (spectra,)
    if length <= 2048:  # (beyond, some launch of few partners is no short one)
        assert check("one_to_many", 1, 2, ls, rs, "f32")["spectra"] == 0


@pytest.mark.parametrize("dtype,mode,n,m,ls,rs,spectra,lefts,partners", [
    # chunks of partners, left spectra first; of one left's partners; of lefts
    ("f32", "one_to_many", 1, 39, (75, 108), (304, 181), 1, 1, 20),
    ("f64", "one_to_many", 1, 55, (44, 167), (147, 167), 1, 1, 28),
    ("f64", "n_to_mn", 3, 21, (53, 196), (307, 141), 1, 3, 4),
    ("f32", "n_to_m", 2, 28, (259, 26), (259, 26), 2, 1, 14),
    ("f32", "n_to_m", 5, 9, (230, 97), (230, 97), 2, 3, 9),
    ("f64", "n_to_m", 5, 35, (81, 160), (81, 160), 2, 3, 35),
])
def test_chunks(dtype, mode, n, m, ls, rs, spectra, lefts, partners):
    form = check(mode, n, m, ls, rs, dtype)
    assert (form["spectra"], form["lefts"], form["partners"]) == (spectra, lefts, partners)


@pytest.mark.parametrize("dtype,mode,n,m,ls,rs", [
    ("f32", "one_to_many", 1, 98, (232, 26), (232, 26)), ("f32", "one_to_many", 1, 20, (9, 235), (335, 21)),
    ("f64", "one_to_many", 1, 10, (13, 396), (377, 22)), ("f64", "n_to_mn", 5, 30, (13, 22), (433, 72)),
    ("f32", "n_to_mn", 6, 12, (212, 212), (212, 212)), ("f32", "one_to_many", 1, 3000, (9, 9), (8, 8)),
])
def test_groups_of_partners_fill_the_gpu(dtype, mode, n, m, ls, rs):
    """Where no spectra are made first (here: no room for them), a group of
    partners shares a left block's transform: no longer groups than leave one
    unit, of at most 128 threads, to every two SMs."""
    form = check(mode, n, m, ls, rs, dtype)
    assert form["spectra"] == 0
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert form["group"] == 1 or form["units"] >= sms // 2
