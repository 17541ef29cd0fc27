"""Buffers that a context makes on first use, where the device has no room for
them: the call reports it, keeps nothing of the attempt, can be made again,
and works once there is room."""

import numpy as np
import pytest
import torch

import amr_oracle as oracle
from test_small_brick_ghosts_gpu import random_state
from test_solve_memory_gpu import MB, only

LEVEL = [0] + [1] * 8
LOC = [(0, 0, 0)] + [(c & 1, (c >> 1) & 1, c >> 2) for c in range(8)]


def context(gpu, physics, max_bricks):
    T = oracle.Tree(LEVEL, LOC, bw=2, nx=8)
    a = gpu.AMR(physics=physics, max_bricks=max_bricks, max_refine_level=1, grid_dim=0.5, z_reflect=0)
    a.load_tree(LEVEL, LOC)
    a.upload_state(random_state(T.n, T.gnx, 2, 21))
    a.enforce_boundaries()
    a.store()
    return a, a.max_dt()


def no_room(gpu, free, call):
    for _ in range(2):
        with pytest.raises(gpu.AmrError) as e:
            call()
        assert e.value.code == -2
        assert free - torch.cuda.mem_get_info()[0] < 32 * MB


@pytest.mark.gpu
@pytest.mark.parametrize("leave", [400 * MB, 760 * MB])  # of 680 MB of state and 151 MB of faces
def test_fused_substep(gpu, leave):
    b, dt = context(gpu, gpu.PHYSICS_EULER, 16)
    b.sub_step(dt, 1.0)
    want = b.download_state()
    b.close()
    a, _ = context(gpu, gpu.PHYSICS_EULER, 8192)
    with only(leave) as free:
        no_room(gpu, free, lambda: a.fused_sub_step(dt, 1.0))
    a.fused_sub_step(dt, 1.0)
    s = (slice(None), slice(None)) + (slice(2, -2),) * 3
    assert np.array_equal(a.download_state()[s], want[s])
    a.close()


@pytest.mark.gpu
def test_poisson(gpu):
    a, _ = context(gpu, gpu.PHYSICS_EULER_GRAVITY, 16384)
    with only(40 * MB) as free:  # of 79 MB of domain-face potential
        no_room(gpu, free, lambda: a.poisson_boundaries())
    a.poisson_solve(1.0e-4)
    b, _ = context(gpu, gpu.PHYSICS_EULER_GRAVITY, 16)
    b.poisson_solve(1.0e-4)
    assert np.array_equal(a.download_poisson(), b.download_poisson())
    a.close()
    b.close()
