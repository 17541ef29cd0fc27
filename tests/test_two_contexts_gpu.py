"""Two contexts used from two host threads at once: plain solves (one
cooperative launch each, on the context's own stream) beside one another and
beside the hydro substeps of a third context give what they give alone."""

import threading

import numpy as np
import pytest

import amr_oracle as oracle
from test_resident_loop_gpu import star
from test_small_brick_ghosts_gpu import random_state

SOLVES = 4


def solves(a, P0, out):
    for _ in range(SOLVES):
        a.upload_poisson(P0)
        out.append(a.poisson_solve(1.0e-5) + (a.download_poisson()[0],))


def hydro(a, U, dt, out):
    for _ in range(SOLVES):
        a.upload_state(U)
        a.enforce_boundaries()
        a.store()
        for _ in range(20):
            a.sub_step(dt, 1.0)
            a.inject_from_children()
        out.append(a.download_state())


@pytest.mark.gpu
def test_threads(gpu):
    stars = [star(gpu, 0, 0)[0] for _ in range(2)]
    P0 = stars[0].download_poisson()
    level = [0] + [1] * 8
    loc = [(0, 0, 0)] + [(c & 1, (c >> 1) & 1, c >> 2) for c in range(8)]
    T = oracle.Tree(level, loc, bw=2, nx=8)
    h = gpu.AMR(physics=gpu.PHYSICS_EULER, max_bricks=16, max_refine_level=1, grid_dim=0.5, z_reflect=0)
    h.load_tree(level, loc)
    U = random_state(T.n, T.gnx, 2, 8)
    h.upload_state(U)
    h.enforce_boundaries()
    dt = 0.1 * h.max_dt()
    alone, alone_h = [], []
    solves(stars[0], P0, alone)
    hydro(h, U, dt, alone_h)
    got = [[], [], []]
    ts = [threading.Thread(target=solves, args=(stars[k], P0, got[k])) for k in range(2)]
    ts.append(threading.Thread(target=hydro, args=(h, U, dt, got[2])))
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k in range(2):
        assert len(got[k]) == SOLVES
        for x, y in zip(got[k], alone):
            assert x[:2] == y[:2] and np.array_equal(x[2], y[2])
    assert len(got[2]) == SOLVES
    for x, y in zip(got[2], alone_h):
        assert np.array_equal(x, y)
    for a in stars + [h]:
        a.close()
