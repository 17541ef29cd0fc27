"""The integer sum that decides most Jacobi sweeps (relax_brick.cuh), emulated
in numpy with its FP32 roundings: whenever it is above RELAX_CLEARLY_ABOVE,
the FP64 sum of squares is above half of the first sweep's.

The bound is the one derived beside the constant: q stands for
2^30 resid / resid0; its relative error is below 16 x 2^-24, and it loses
less than one unit for each of the at most 864 threads, so a margin of 4096
units above 2^29 leaves no room for a disagreement.  Sums are placed at the
threshold and a few margins around it, with cells of like and of very
different sizes, over the range of resid0 that takes this path."""

import numpy as np
import pytest

CLEARLY_ABOVE = (1 << 29) + 4096


def integer_sum(tmp0, resid0, threads, ct):
    """tmp0: [K, threads] values in the correction's type."""
    s = np.float32(32768.0) * (np.float32(1.0) / np.sqrt(np.float32(resid0)))
    t = tmp0.astype(ct).astype(np.float32) * s
    f = np.zeros(threads, np.float32)
    for r in range(t.shape[0]):
        f = f + t[r] * t[r]
    return int(np.trunc(f).astype(np.uint64).sum())


@pytest.mark.parametrize("threads,k", [(512, 1), (256, 2), (576, 3), (864, 2), (288, 6)])
@pytest.mark.parametrize("ct", [np.float32, np.float64])
def test_clear_answers_are_the_fp64_sums(threads, k, ct):
    rng = np.random.default_rng(threads + k)
    clear = 0
    for trial in range(400):
        resid0 = 10.0 ** rng.uniform(-30.0, 30.0)
        spread = rng.choice([0.0, 1.0, 6.0])
        v = rng.standard_normal((k, threads)) * 10.0 ** rng.uniform(-spread, 0.0, (k, threads))
        # the sum lands within a few margins (4096 / 2^29 = 7.6e-6) of half of resid0
        want = 0.5 * resid0 * (1.0 + rng.uniform(-4e-5, 4e-5))
        v = (v * np.sqrt(want / (v * v).sum())).astype(ct)
        resid = (v.astype(np.float64) ** 2).sum()
        q = integer_sum(v, resid0, threads, ct)
        assert q < 1 << 31
        if q > CLEARLY_ABOVE:
            clear += 1
            assert resid > 0.5 * resid0, (trial, q, resid / resid0)
        else:
            # no needless FP64 sum far from the threshold
            assert resid < 0.5 * resid0 * (1.0 + 4.0 * 4096.0 / (1 << 29)), (trial, q, resid / resid0)
    assert clear > 50
