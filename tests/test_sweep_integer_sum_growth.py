"""The integer sum that decides most Jacobi sweeps (relax_brick.cuh), emulated
with its FP32 roundings and its 32-bit sums and the constants read from the
header: a clear answer, either way, is the FP64 sums' for any ratio of a
sweep's sum to the first one's -- near one half, and also far above it, where
a 32-bit sum must not wrap (at rounding level a sweep's sum can grow).

The bound is the one derived beside the constants: relative errors below
36 x 2^-24, and less than one unit lost for each of at most 864 threads."""

import os
import re

import numpy as np
import pytest

from conftest import PKG

HEADER = open(os.path.join(PKG, "csrc", "relax_brick.cuh")).read()
SCALE = np.float32(re.search(r"RELAX_SCALE = ([0-9.]+)f;", HEADER).group(1))
HALF = 1 << int(re.search(r"RELAX_HALF = 1u << (\d+)", HEADER).group(1))
MARGIN = int(re.search(r"RELAX_MARGIN = (\d+)u", HEADER).group(1))
ABOVE, BELOW = HALF + MARGIN, HALF - MARGIN


def tree_sum(v):
    """FP32 butterfly sums of warps, then of the warps' sums."""
    v = np.concatenate([v, np.zeros(-len(v) % 32, np.float32)]).reshape(-1, 32)
    while v.shape[1] > 1:
        v = v[:, ::2] + v[:, 1::2]
    return v[0, 0] if v.shape[0] == 1 else tree_sum(v[:, 0])


def thread_sums(t):
    f = np.zeros(t.shape[1], np.float32)
    for r in range(t.shape[0]):
        f = f + t[r] * t[r]
    return f


def integer_sum(first, tmp0):
    r0 = tree_sum(thread_sums(first.astype(np.float32)))
    s = SCALE * (np.float32(1.0) / np.sqrt(r0))
    with np.errstate(over="ignore"):
        f = thread_sums(tmp0.astype(np.float32) * s)
    u = np.trunc(np.minimum(f, np.float32(ABOVE + 1))).astype(np.uint64)
    q = int(u.sum())
    assert q < 1 << 32  # so no order of 32-bit sums wraps
    return q


def values(rng, k, threads, total, ct):
    """k x threads values whose squares add up to `total`: alike, of very
    different sizes, or all in one cell."""
    spread = rng.choice([0.0, 1.0, 6.0])
    v = rng.standard_normal((k, threads)) * 10.0 ** rng.uniform(-spread, 0.0, (k, threads))
    if rng.random() < 0.2:
        one = np.zeros_like(v)
        one[rng.integers(k), rng.integers(threads)] = 1.0
        v = one
    return (v * np.sqrt(total / (v * v).sum())).astype(ct)


def test_constants():
    assert SCALE * SCALE == 2 * HALF
    assert MARGIN > 864 + 36 * 2.0 ** -24 * HALF + 1
    assert 864 * (ABOVE + 1) < 1 << 32
    assert "K <= 6 && TH <= 864" in HEADER


@pytest.mark.parametrize("threads,k", [(512, 1), (256, 2), (576, 3), (864, 2), (288, 6)])
@pytest.mark.parametrize("ct", [np.float32, np.float64])
@pytest.mark.parametrize("ratios", ["at the threshold", "below one", "grown"])
def test_clear_answers_are_the_fp64_sums(threads, k, ct, ratios):
    rng = np.random.default_rng(threads + k)
    clear = 0
    for trial in range(300):
        resid0 = 10.0 ** rng.uniform(-27.5, 27.5)
        if ratios == "at the threshold":
            ratio = 0.5 * (1.0 + rng.uniform(-4.0, 4.0) * MARGIN / HALF)
        elif ratios == "below one":
            ratio = rng.uniform(0.0, 1.0)
        else:
            ratio = 10.0 ** rng.uniform(0.0, 6.0)
        first = values(rng, k, threads, resid0, ct)
        tmp0 = values(rng, k, threads, ratio * resid0, ct)
        q = integer_sum(first, tmp0)
        exact0 = (first.astype(np.float64) ** 2).sum()
        exact = (tmp0.astype(np.float64) ** 2).sum()
        if q > ABOVE:
            assert exact > 0.5 * exact0, (trial, q, exact / exact0)
        elif q < BELOW:
            assert exact < 0.5 * exact0, (trial, q, exact / exact0)
        clear += q > ABOVE or q < BELOW
        # no needless FP64 sum far from the threshold
        if abs(exact / exact0 - 0.5) > 2.0 * MARGIN / HALF:
            assert q > ABOVE or q < BELOW, (trial, q, exact / exact0)
    assert clear > 100
