"""A tree with more bricks than the context's pool: the call that makes it and
every device call after it are refused with AMR_ERR_CAPACITY, and a tree that
fits brings the context back."""

import numpy as np
import pytest

import amr_oracle as oracle
from test_small_brick_ghosts_gpu import random_state

LEVEL = [0] + [1] * 8
LOC = [(0, 0, 0)] + [(c & 1, (c >> 1) & 1, c >> 2) for c in range(8)]


def one_step(a, T):
    a.upload_state(random_state(T.n, T.gnx, T.bw, 11))
    a.enforce_boundaries()
    dt = a.max_dt()
    a.store()
    a.sub_step(dt, 1.0)
    a.inject_from_children()
    a.enforce_boundaries()
    return dt, a.download_state(), a.flow_off()


def refused(gpu, call):
    with pytest.raises(gpu.AmrError) as e:
        call()
    assert e.value.code == -7, e.value


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["load", "refine"])
def test_more_bricks_than_the_pool(gpu, how):
    T = oracle.Tree(LEVEL, LOC, bw=2, nx=8)
    cfg = dict(physics=gpu.PHYSICS_EULER_GRAVITY, max_refine_level=2, grid_dim=0.5, z_reflect=0, mirror_refine_y=0)
    b = gpu.AMR(max_bricks=32, **cfg)
    b.load_tree(LEVEL, LOC)
    want = one_step(b, T)
    b.close()
    a = gpu.AMR(max_bricks=9, **cfg)
    a.load_tree(LEVEL, LOC)
    one_step(a, T)
    a.set_flow_off(np.zeros(a.nf))
    if how == "load":
        refused(gpu, lambda: a.load_tree(LEVEL + [2], LOC + [(2, 2, 2)]))
        assert a.nbricks == 10
    else:
        flags = np.zeros((9, 8), np.uint8)
        flags[0] = 1
        flags[1, 7] = 1
        refused(gpu, lambda: a.refine_from_flags(flags))
        assert a.nbricks > 9
    n = a.get_tree()["level"].size
    assert n == a.nbricks
    for call in (a.enforce_boundaries, a.compute_fluxes, a.max_dt, a.store, a.download_state, a.inject_from_children,
                 a.poisson_boundaries, a.compute_forces, a.vcycle, lambda: a.sub_step(1e-3, 1.0),
                 lambda: a.poisson_solve(1e-3), lambda: a.graph_solve(1e-3), lambda: a.check_for_refine(1.0),
                 lambda: a.fused_sub_step(1e-3, 1.0), lambda: a.state_max(0), lambda: a.state_sum(0)):
        refused(gpu, call)
    a.load_tree(LEVEL, LOC)
    a.set_flow_off(np.zeros(a.nf))
    got = one_step(a, T)
    assert got[0] == want[0] and np.array_equal(got[2], want[2])
    s = (slice(None), slice(None)) + (slice(2, -2),) * 3
    assert np.array_equal(got[1][s], want[1][s])
    a.close()
