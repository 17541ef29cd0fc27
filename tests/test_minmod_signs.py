"""minmod2 as the device forms it (one compare and the sign bits,
euler_state.cuh), restated in numpy, against the reference's formula
0.5 (sgn(a) + sgn(b)) min(|a|, |b|) (real.h:63-65): equal values for every pair
of a grid of ordinary, tiny, huge and special numbers (zeros may differ in
sign)."""

import numpy as np
import pytest


def reference(a, b):
    sgn = lambda x: np.where(x > 0, 1.0, np.where(x < 0, -1.0, 0.0)).astype(a.dtype)
    fa, fb = np.abs(a), np.abs(b)
    return a.dtype.type(0.5) * (sgn(a) + sgn(b)) * np.where(fa > fb, fb, fa)


def device(a, b):
    fa, fb = np.abs(a), np.abs(b)
    m = np.where(fa > fb, fb, fa)
    r = np.where(np.signbit(a) != np.signbit(b), m - m, np.copysign(m, a))
    return np.where(np.isnan(b), a * a.dtype.type(0.5), r)


@pytest.mark.parametrize("dt", [np.float64, np.float32])
def test_same_values(dt):
    rng = np.random.default_rng(3)
    f = np.finfo(dt)
    v = [0.0, f.tiny, f.smallest_subnormal, 1.0, 1.0 + f.eps, 0.75, 1e10, f.max, np.inf, np.nan]
    v = np.array(v + [-x for x in v] + list(rng.standard_normal(200) * 10.0 ** rng.uniform(-30, 30, 200)), dt)
    a, b = np.meshgrid(v, v)
    with np.errstate(all="ignore"):
        x, y = device(a, b), reference(a, b)
    assert np.array_equal(x, y, equal_nan=True)
