"""The fused FFT kernels (normalised results of the FFT method) against the
oracle, at the edges of their dispatch: every transform length, sizes one
below and one above a length, single rows and columns, odd row counts (a row
pair with one row), partner counts that leave partial groups and chunks, and
sizes beyond the kernels' lengths, which keep the library transforms.

Bounds: those of the FFT path elsewhere, 1e-5 of max|oracle| for FP32 and
1e-10 for FP64 (an FFT's error is a few roundings per pass, below 1e-6 and
1e-14 of the result's scale at these sizes).
"""
import numpy as np
import pytest

from helpers import rel_to_max, seeded
from oracle import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import xcorr  # noqa: E402

LENGTHS = [16, 32, 48, 64, 80, 96, 112, 128, 160, 192, 224, 256, 320, 384, 448, 512, 640, 768, 896, 1024, 1280, 1536,
           1792, 2048, 2560, 3072, 3584, 4096]
TOL = {"f32": 1e-5, "f64": 1e-10}


def run(mode, left, right, dtype):
    l, r = torch.from_numpy(left).cuda(), torch.from_numpy(right).cuda()
    n_out = xcorr.output_count(mode, left.shape[0], right.shape[0])
    out = torch.full((n_out, left.shape[1] + right.shape[1] - 1, left.shape[2] + right.shape[2] - 1), float("nan"),
                     dtype=l.dtype, device="cuda")
    xcorr.correlate(mode, l, r, method="fft", out=out)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def check(mode, n, m, ls, rs, dtype, dist="signed", seed=5):
    npdt = np.float32 if dtype == "f32" else np.float64
    left, right = seeded((n,) + ls, seed, dist, npdt), seeded((m,) + rs, seed + 1, dist, npdt)
    ref = oracle.run_mode(mode, left, right, dtype="f32acc64" if dtype == "f32" else "f64", threads=8)
    assert rel_to_max(run(mode, left, right, dtype), ref) <= TOL[dtype]


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("n", LENGTHS)
def test_every_length_as_rows_and_columns(n, dtype):
    """Full output size exactly n (no slack) and n - 1 on either axis."""
    thin = 3
    check("one_to_one", 1, 1, (thin, n - n // 3), (4, n // 3 + 1), dtype)
    check("one_to_one", 1, 1, (n - n // 3, thin), (n // 3, 4), dtype)


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("mode,n,m", [("one_to_one", 1, 1), ("one_to_many", 1, 11), ("n_to_mn", 3, 21),
                                      ("n_to_m", 5, 7), ("n_to_m", 4, 1)])
@pytest.mark.parametrize("ls,rs", [((1, 1), (1, 1)), ((1, 40), (1, 25)), ((40, 1), (25, 1)), ((33, 20), (16, 45)),
                                   ((64, 64), (64, 64)), ((17, 70), (80, 3))])
def test_modes_and_ragged_sizes(mode, n, m, ls, rs, dtype):
    check(mode, n, m, ls, rs, dtype, "normal")


def check_against_stages(mode, n, m, ls, rs, dtype):
    """The fused result against the library transforms run stage by stage."""
    npdt = np.float32 if dtype == "f32" else np.float64
    left = torch.from_numpy(seeded((n,) + ls, 7, "uniform", npdt)).cuda()
    right = torch.from_numpy(seeded((m,) + rs, 8, "uniform", npdt)).cuda()
    plan = xcorr.FftPlan(mode, dtype, ls, n, rs, m)
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


@pytest.mark.parametrize("mode,n,m", [("one_to_many", 1, 45), ("n_to_mn", 2, 50), ("n_to_m", 3, 17)])
def test_many_partners(mode, n, m):
    """More partners than a launch has waves: the column kernels' dense form."""
    check_against_stages(mode, n, m, (400, 380), (390, 400), "f32")


@pytest.mark.parametrize("dtype", ["f32", "f64"])
@pytest.mark.parametrize("mode,n,m", [("one_to_one", 1, 1), ("one_to_many", 1, 2), ("n_to_mn", 2, 6)])
@pytest.mark.parametrize("size", [320, 530, 700, 1000, 1100, 1300, 1900])
def test_few_large_partners(size, mode, n, m, dtype):
    """Either side of the rule for making the left spectra first, and sizes
    whose workspace has no room for them (lengths rounded up by much)."""
    check_against_stages(mode, n, m, (size, size), (size, size), dtype)
    check_against_stages(mode, n, m, (size, size - 7), (size - 30, size // 2), dtype)


def test_beyond_the_kernels_lengths():
    check("one_to_one", 1, 1, (2, 3000), (3, 1200), "f32")
