"""The Newton inversion whose lanes take the next point of their warp's run:
every point's temperature, iterations and status, whatever the number of
points (a part of a warp, a warp, runs of more than a warp's points) and
whatever the neighbours of a point do (floor temperature, many iterations,
outside the table): the same as in calls of a warp's points at most."""

import numpy as np
import pytest

from conftest import _load_pkg_module


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 31, 33, 127, 56_833, 300_001])
@pytest.mark.parametrize("from_entropy", [False, True])
def test_every_point_is_its_own(gpu, table_path, n, from_entropy):
    h = _load_pkg_module("helm_b200", "helm.py").Helm(table_path)
    rng = np.random.default_rng(n)
    rho = 10.0 ** rng.uniform(-2.0, 9.0, n)
    T = 10.0 ** rng.uniform(4.0, 9.0, n)
    abar = rng.uniform(12.0, 16.0, n)
    f = h.eos(rho, T, abar, abar / 2.0)
    target = (f["s"] if from_entropy else f["e"]).copy()
    target[::7] *= 0.5          # below the floor's value for many of these
    rho[3::11] = 1.0e40         # outside the table
    guess = T * 10.0 ** rng.uniform(-1.5, 1.5, n)
    got = h.invert_T(rho, target, abar, abar / 2.0, guess, from_entropy=from_entropy)
    # a sample of the points, in calls of one warp's points at most
    pick = np.unique(np.concatenate([np.arange(min(n, 40)), rng.integers(0, n, 60), [n - 1]]))
    for a in range(0, pick.size, 32):
        q = pick[a:a + 32]
        one = h.invert_T(rho[q], target[q], abar[q], abar[q] / 2.0, guess[q], from_entropy=from_entropy)
        for k in ("T", "iters", "status"):
            assert np.array_equal(got[k][q], one[k]), k
        inside = one["status"] != 1  # outside the table the other outputs are undefined
        for k in ("p", "e", "cs", "cv", "s"):
            assert np.array_equal(got[k][q][inside], one[k][inside], equal_nan=True), k
    out = got["status"] == 1
    assert np.all(out[3::11]) and np.array_equal(got["T"][3::11], guess[3::11])
    h.close()
