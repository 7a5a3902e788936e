"""Ragged plans' routed pairs through the fused FFT kernels: several chunks of
spectra, outputs beyond the kernels' lengths beside ordinary ones, thin and
odd matrices, and values near the ends of the FP32 range."""
import numpy as np
import pytest

from helpers import rel_to_max
from oracle import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import xcorr  # noqa: E402


def routed(plan):
    """The variant that routes the most pairs (tile shape 0)."""
    n = plan.describe()["n_variants"]
    plan.select(n - 2)
    return plan.describe()["tc_pairs"]


def run(plan):
    plan.out.fill_(float("nan"))
    plan.execute()
    torch.cuda.synchronize()
    return plan.outputs()


def test_several_chunks_match_single_calls():
    """40 pairs of 1400x1300 with 601x700: about 1.6 GiB of spectra, more than
    one chunk (1 GiB) holds; each against one FFT call of the pair."""
    rng = np.random.default_rng(21)
    lefts = [rng.random((1400, 1300), dtype=np.float32) for _ in range(5)]
    rights = [rng.random((601, 700), dtype=np.float32) for _ in range(8)]
    pairs = [(a, b) for a in range(5) for b in range(8)]
    plan = xcorr.RaggedPlan(lefts, rights, pairs)
    assert routed(plan) == 40
    outs = run(plan)
    for (a, b), got in zip(pairs, outs):
        ref = xcorr.correlate("one_to_one", torch.from_numpy(lefts[a]).cuda(), torch.from_numpy(rights[b]).cuda(),
                              method="fft")[0].cpu().numpy()
        # two evaluations of the same transforms, below 1e-6 from the exact result each
        assert rel_to_max(got, ref) <= 2e-6
    plan.close()


def test_mixed_engines_match_oracle():
    """A strip whose output is wider than the longest transform stays on the
    split-BF16 path, beside FFT pairs of odd and thin shapes and small pairs
    on the plain kernel.  Tolerance: the accuracy gate, 1e-5."""
    rng = np.random.default_rng(22)
    sides = [(4, 3000, 4, 2000), (3, 2100, 9, 1990), (257, 31, 129, 255), (1500, 40, 40, 30), (20, 20, 20, 20),
             (511, 65, 33, 64)]
    lefts = [rng.uniform(-1, 1, (a, b)).astype(np.float32) for a, b, _, _ in sides]
    rights = [rng.uniform(-1, 1, (c, d)).astype(np.float32) for _, _, c, d in sides]
    pairs = [(i, i) for i in range(len(sides))]
    plan = xcorr.RaggedPlan(lefts, rights, pairs)
    assert routed(plan) == 5
    for got, ref in zip(run(plan), oracle.run_pairs(lefts, rights, threads=8)):
        assert rel_to_max(got, ref) <= 1e-5
    plan.close()


@pytest.mark.parametrize("exponent", [-50, 55])
def test_results_near_the_ends_of_the_range(exponent):
    """Inputs scaled by a power of two give the scaled result while it is in
    FP32 range (products of 2^-100, and of 2^110 times the 2^16 sums), within
    the FFT's rounding of two differently scaled runs."""
    rng = np.random.default_rng(23)
    left = rng.uniform(-1, 1, (300, 280)).astype(np.float32)
    right = rng.uniform(-1, 1, (290, 270)).astype(np.float32)
    got = []
    for e in (0, exponent):
        plan = xcorr.RaggedPlan([np.ldexp(left, e)], [np.ldexp(right, e)], [(0, 0)])
        assert routed(plan) == 1
        got.append(run(plan)[0].astype(np.float64))
        plan.close()
    assert np.isfinite(got[1]).all()
    assert rel_to_max(np.ldexp(got[1], -2 * exponent), got[0]) <= 1e-6
