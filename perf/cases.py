"""Performance cases of the cross-correlation library.

Each case is one call (or one plan replay) that a program using the library
makes through its public Python entry points: ``xcorr.correlate`` with a
method name, ``xcorr.FftPlan`` and ``xcorr.RaggedPlan``.  Sizes, distributions
and batch forms are those of the library's own benchmark and tests, plus
generic odd ones.  ``draw`` spreads further cases over the same ranges.
"""
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PKG = os.path.join(_ROOT, "cross-corr_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import xcorr  # noqa: E402

_TORCH = {"f32": torch.float32, "f64": torch.float64}


def _dense(name, mode, method, n, left, m, right, dist, dtype="f32", plan=False):
    c = {"kind": "dense", "mode": mode, "method": method, "dtype": dtype, "dist": dist, "n": n, "hl": left[0],
         "wl": left[1], "m": m, "hr": right[0], "wr": right[1], "plan": plan}
    return dict(c, name=name) if name else c


def _ragged(name, pairs, lo, hi, shapes):
    c = {"kind": "ragged", "pairs": pairs, "lo": lo, "hi": hi, "shapes": shapes, "dtype": "f32", "dist": "signed"}
    return dict(c, name=name) if name else c


def listed():
    return [
        # One small pair with the library choosing the algorithm: the call a
        # program makes per object or per feature, where latency counts.
        _dense("pair_32_auto", "one_to_one", "auto", 1, (32, 32), 1, (32, 32), "uniform"),
        # One pair of 128x128 matrices by the definition: the benchmark's
        # smallest configuration.
        _dense("pair_128_direct", "one_to_one", "direct", 1, (128, 128), 1, (128, 128), "uniform"),
        # One image against 64 candidates by the definition in plain FP32: the
        # benchmark's headline inputs on the default method.
        _dense("batch_256_direct", "one_to_many", "direct", 1, (256, 256), 64, (256, 256), "uniform"),
        # A few images against a few smaller patches, odd sizes whose rows are
        # not 16-byte aligned.
        _dense("odd_patches_direct", "n_to_m", "direct", 3, (201, 183), 6, (75, 59), "signed"),
        # FP64 by the definition (the command line's `-d double`), 8 left
        # matrices each with its own 4 partners.
        _dense("n_to_mn_64_f64_direct", "n_to_mn", "direct", 8, (64, 64), 32, (64, 64), "normal", "f64"),
        # The headline workload on the split-BF16 tensor-core path.
        _dense("batch_256_bf16x3", "one_to_many", "tc_bf16x3", 1, (256, 256), 64, (256, 256), "uniform"),
        # Many small zero-mean pairs on the split-BF16 path: 8 x 32 matrices,
        # 256 outputs.
        _dense("n_to_m_64_bf16x3", "n_to_m", "tc_bf16x3", 8, (64, 64), 32, (64, 64), "normal"),
        # Template search: 16 small templates over a large image, split TF32.
        _dense("templates_1024_tf32x3", "one_to_many", "tc_tf32x3", 1, (1024, 1024), 16, (32, 32), "uniform"),
        # The headline inputs through the FFT path, the fastest for most
        # problems and what the selector picks.
        _dense("batch_256_fft", "one_to_many", "fft", 1, (256, 256), 64, (256, 256), "uniform"),
        # Large images through an explicit FFT plan: 2048x2048, 16 partners.
        _dense("large_2048_fft_plan", "one_to_many", "fft", 1, (2048, 2048), 16, (2048, 2048), "uniform", plan=True),
        # Every pair of small FP64 matrices through the FFT path.
        _dense("n_to_m_64_f64_fft", "n_to_m", "fft", 8, (64, 64), 32, (64, 64), "normal", "f64"),
        # Pairs of uneven sizes as one autotuned plan, replayed.
        _ragged("ragged_96", 96, 16, 512, 4),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case: any method, mode and type over the listed sizes."""
    kind = rng.choice(["auto", "direct", "direct", "direct", "f64_direct", "tc", "tc", "fft", "fft", "fft", "f64_fft",
                       "ragged"])
    if kind == "ragged":
        lo = rng.randint(8, 64)
        return _ragged(None, rng.randint(24, 96), lo, rng.randint(max(96, 2 * lo), 512), rng.randint(0, 10 ** 6))
    method = {"auto": "auto", "direct": "direct", "f64_direct": "direct", "fft": "fft", "f64_fft": "fft"}.get(
        kind, rng.choice(["tc_bf16x3", "tc_bf16x3", "tc_tf32x3"]))
    dtype = "f64" if kind.startswith("f64") else "f32"
    # a pass costs no more than the largest listed one of its kind: multiply-
    # adds where the method counts them, output elements for FFT
    macs = {"auto": 2e9, "direct": 1.3e11, "f64_direct": 1e9, "tc": 2.5e11}.get(kind, 1e15)
    elems = {"fft": 1.2e8, "f64_fft": 8e6}.get(kind, 1e8)
    hi = {"auto": 256, "direct": 512, "f64_direct": 160, "tc": 1024, "fft": 2048, "f64_fft": 256}[kind]
    while True:
        mode = rng.choice(["one_to_one", "one_to_many", "n_to_mn", "n_to_m"])
        n = 1 if mode.startswith("one") else rng.randint(2, 8)
        m = {"one_to_one": 1, "one_to_many": _log_int(rng, 2, 128), "n_to_mn": n * rng.randint(1, 8),
             "n_to_m": rng.randint(2, 32)}[mode]
        hl, wl = _log_int(rng, 16, hi), _log_int(rng, 16, hi)
        form = rng.choice(["equal", "equal", "template", "any"])
        if form == "equal":  # square inputs are the most common; equal sizes next
            if rng.random() < 0.5:
                wl = hl
            hr, wr = hl, wl
        elif form == "template":
            hr, wr = _log_int(rng, 8, max(8, hl // 2)), _log_int(rng, 8, max(8, wl // 2))
        else:
            hr, wr = _log_int(rng, 16, hi), _log_int(rng, 16, hi)
        n_out = n * m if mode == "n_to_m" else m
        if n_out * hl * wl * hr * wr <= macs and n_out * (hl + hr) * (wl + wr) <= elems:
            break
    return _dense(None, mode, method, n, (hl, wl), m, (hr, wr), rng.choice(["uniform", "normal", "signed"]), dtype,
                  plan=method == "fft" and rng.random() < 0.4)


def _values(gen, shape, dist, dtype):
    if dist == "normal":
        return torch.randn(shape, generator=gen, dtype=dtype, device="cuda")
    x = torch.rand(shape, generator=gen, dtype=dtype, device="cuda")
    return x * 2 - 1 if dist == "signed" else x


def _inputs(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    dt = _TORCH[case["dtype"]]
    return (_values(gen, (case["n"], case["hl"], case["wl"]), case["dist"], dt),
            _values(gen, (case["m"], case["hr"], case["wr"]), case["dist"], dt))


def _ragged_inputs(case, seed):
    """Pair sizes come from the case (a program's batch keeps its shapes),
    values from the seed."""
    rs = np.random.default_rng(case["shapes"])
    sizes = rs.integers(case["lo"], case["hi"] + 1, size=(case["pairs"], 4))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    flat = _values(gen, (int((sizes[:, 0] * sizes[:, 1]).sum() + (sizes[:, 2] * sizes[:, 3]).sum()),), case["dist"],
                   torch.float32).cpu().numpy()
    lefts, rights, off = [], [], 0
    for hl, wl, hr, wr in sizes.tolist():
        lefts.append(flat[off:off + hl * wl].reshape(hl, wl))
        off += hl * wl
        rights.append(flat[off:off + hr * wr].reshape(hr, wr))
        off += hr * wr
    return lefts, rights


def _n_out(case):
    return xcorr.output_count(case["mode"], case["n"], case["m"])


def prepare(case, seed):
    if case["kind"] == "ragged":
        lefts, rights = _ragged_inputs(case, seed)
        plan = xcorr.RaggedPlan(lefts, rights, [(i, i) for i in range(len(lefts))])
        plan.autotune()
        return {"ragged": plan}
    left, right = _inputs(case, seed)
    out = torch.empty((_n_out(case), case["hl"] + case["hr"] - 1, case["wl"] + case["wr"] - 1), dtype=left.dtype,
                      device="cuda")
    state = {"mode": case["mode"], "method": case["method"], "left": left, "right": right, "out": out, "plan": None}
    shapes = ((case["hl"], case["wl"]), case["n"], (case["hr"], case["wr"]), case["m"])
    if case["plan"]:
        state["plan"] = xcorr.FftPlan(case["mode"], case["dtype"], *shapes)
        ws = state["plan"].workspace_bytes
    else:
        ws = xcorr.workspace_size(case["mode"], case["dtype"], case["method"], *shapes)
    state["ws"] = torch.empty(max(1, ws), dtype=torch.uint8, device="cuda")
    return state


def run(state):
    if "ragged" in state:
        state["ragged"].execute()
        return state["ragged"].out
    if state["plan"] is not None:
        return state["plan"].execute(state["left"], state["right"], state["out"], state["ws"])
    return xcorr.correlate(state["mode"], state["left"], state["right"], method=state["method"], out=state["out"],
                           workspace=state["ws"])


def _fft_flops(hl, wl, hr, wr, n_in, n_out):
    """Real transforms of the full output size (2.5 N log2 N each) and one
    complex product per bin and output."""
    n = (hl + hr - 1) * (wl + wr - 1)
    return 2.5 * n * math.log2(max(2, n)) * (n_in + n_out) + 3.0 * n * n_out


def work(case):
    if case["kind"] == "ragged":
        rs = np.random.default_rng(case["shapes"])
        b = f = 0.0
        for hl, wl, hr, wr in rs.integers(case["lo"], case["hi"] + 1, size=(case["pairs"], 4)).tolist():
            b += 4.0 * (hl * wl + hr * wr + (hl + hr - 1) * (wl + wr - 1))
            f += min(2.0 * hl * wl * hr * wr, _fft_flops(hl, wl, hr, wr, 2, 1))
        return {"bytes": b, "flops": f}
    hl, wl, hr, wr, n, m = (case[k] for k in ("hl", "wl", "hr", "wr", "n", "m"))
    n_out = n * m if case["mode"] == "n_to_m" else m
    es = 8 if case["dtype"] == "f64" else 4
    b = es * (n * hl * wl + m * hr * wr + n_out * (hl + hr - 1) * (wl + wr - 1))
    direct, fft = 2.0 * hl * wl * hr * wr * n_out, _fft_flops(hl, wl, hr, wr, n + m, n_out)
    f = fft if case["method"] == "fft" else min(direct, fft) if case["method"] == "auto" else direct
    return {"bytes": b, "flops": f}


def _exact_pair(lspec, right, shape, crop):
    """out[sy + Hr - 1][sx + Wr - 1] = sum L[y + sy][x + sx] R[y][x], as the
    full convolution with the flipped right matrix."""
    rspec = torch.fft.rfft2(torch.flip(right.double(), (-2, -1)), s=shape)
    return torch.fft.irfft2(lspec * rspec, s=shape)[..., :crop[0], :crop[1]]


def _pow2(n):
    return 1 << max(0, (n - 1).bit_length())


def exact(case, seed):
    if case["kind"] == "ragged":
        lefts, rights = _ragged_inputs(case, seed)
        outs = []
        for a, b in zip(lefts, rights):
            crop = (a.shape[0] + b.shape[0] - 1, a.shape[1] + b.shape[1] - 1)
            shape = (_pow2(crop[0]), _pow2(crop[1]))
            spec = torch.fft.rfft2(torch.from_numpy(a).cuda().double(), s=shape)
            outs.append(_exact_pair(spec, torch.from_numpy(b).cuda(), shape, crop).reshape(-1))
        return torch.cat(outs)
    left, right = _inputs(case, seed)
    n, m = case["n"], case["m"]
    crop = (case["hl"] + case["hr"] - 1, case["wl"] + case["wr"] - 1)
    shape = (_pow2(crop[0]), _pow2(crop[1]))
    if case["mode"] == "n_to_m":
        pairs = [(a, b) for a in range(n) for b in range(m)]
    else:
        pairs = [(b % n, b) for b in range(m)]
    out = torch.empty((len(pairs),) + crop, dtype=torch.float64, device="cuda")
    for a in range(n):
        spec = torch.fft.rfft2(left[a].double(), s=shape)
        for o, (la, b) in enumerate(pairs):
            if la == a:
                out[o] = _exact_pair(spec, right[b], shape, crop)
    return out
