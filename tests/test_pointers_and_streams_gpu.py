"""Calls on buffers that start at any element, on a non-blocking stream right
behind the kernels that make their inputs and in front of those that reuse them,
with one workspace for several problems, and captured into a caller's graph.

Results are compared with the same calls on fresh buffers on the default stream;
two runs of one kernel differ at most by the order of its atomic adds: 2e-6 of
max|out| in FP32 and 1e-14 in FP64."""
import numpy as np
import pytest

from helpers import seeded

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import xcorr  # noqa: E402

TOL = {"f32": 2e-6, "f64": 1e-14}
METHODS = [("direct", "f32"), ("direct", "f64"), ("direct:1", "f32"), ("direct:2", "f64"), ("fft", "f32"), ("fft", "f64"),
           ("tc_bf16x3", "f32"), ("tc_tf32x3", "f32")]
CASES = [
    ("one_to_one", 1, 1, (64, 64), (64, 64)), ("one_to_many", 1, 33, (96, 128), (40, 64)),
    ("n_to_mn", 3, 12, (61, 43), (25, 30)), ("n_to_m", 4, 30, (128, 100), (90, 77)),
]
IDS = [c[0] for c in CASES]


def inputs(case, dtype, seed):
    _, n, m, ls, rs = case
    npdt = np.float32 if dtype == "f32" else np.float64
    return (torch.from_numpy(seeded((n,) + ls, seed, "signed", npdt)).cuda(),
            torch.from_numpy(seeded((m,) + rs, seed + 1, "signed", npdt)).cuda())


def close(a, b, dtype):
    return float((a - b).abs().max()) <= TOL[dtype] * float(b.abs().max())  # (False for a NaN)


def moved(t, offset):
    """The same values `offset` elements into a larger buffer."""
    buf = torch.full((t.numel() + 8,), float("nan"), dtype=t.dtype, device="cuda")
    v = buf[offset:offset + t.numel()].view(t.shape)
    v.copy_(t)
    return buf, v


@pytest.mark.parametrize("method,dtype", METHODS)
@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_any_element_offset(case, method, dtype):
    left, right = inputs(case, dtype, 11)
    ref = xcorr.correlate(case[0], left, right, method=method)
    for ol, orr, oo in ((1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 2, 3), (3, 1, 2)):
        (_, l), (_, r), (buf, out) = moved(left, ol), moved(right, orr), moved(torch.full_like(ref, float("nan")), oo)
        xcorr.correlate(case[0], l, r, method=method, out=out)
        assert close(out, ref, dtype)
        # nothing beside the output is written
        assert torch.isnan(buf[:oo]).all() and torch.isnan(buf[oo + out.numel():]).all()


@pytest.mark.parametrize("method,dtype", METHODS)
@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_behind_a_producer_on_a_side_stream(case, method, dtype):
    """Inputs made, used and overwritten on one stream, the output copied and
    filled anew, one workspace for all: many calls in flight."""
    sets = [inputs(case, dtype, 21 + 2 * i) for i in range(3)]
    refs = [xcorr.correlate(case[0], l, r, method=method).clone() for l, r in sets]
    need = xcorr.workspace_size(case[0], dtype, method.partition(":")[0], case[3], case[1], case[4], case[2])
    ws = torch.empty(max(1, need), dtype=torch.uint8, device="cuda")
    left, right, out = torch.empty_like(sets[0][0]), torch.empty_like(sets[0][1]), torch.empty_like(refs[0])
    kept = [torch.empty_like(refs[0]) for _ in range(9)]
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.Stream()):
        for i in range(9):
            torch.add(sets[i % 3][0], 0, out=left)
            torch.add(sets[i % 3][1], 0, out=right)
            out.fill_(float("nan"))
            xcorr.correlate(case[0], left, right, method=method, out=out, workspace=ws)
            left.fill_(float("nan"))
            right.fill_(float("nan"))
            kept[i].copy_(out)
    torch.cuda.synchronize()
    for i in range(9):
        assert close(kept[i], refs[i % 3], dtype)


@pytest.mark.parametrize("method,dtype", METHODS)
@pytest.mark.parametrize("case", CASES, ids=IDS)
def test_captured_into_a_graph(case, method, dtype):
    left, right = inputs(case, dtype, 31)
    ref = xcorr.correlate(case[0], left, right, method=method)
    need = xcorr.workspace_size(case[0], dtype, method.partition(":")[0], case[3], case[1], case[4], case[2])
    ws = torch.empty(max(1, need), dtype=torch.uint8, device="cuda")
    out, copy = torch.empty_like(ref), torch.empty_like(ref)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(2):
            out.fill_(float("nan"))
            xcorr.correlate(case[0], left, right, method=method, out=out, workspace=ws)
            copy.copy_(out)
    for _ in range(3):
        copy.fill_(0)
        graph.replay()
        torch.cuda.synchronize()
        assert close(copy, ref, dtype)
