"""Bricks above 12^3: the same grid as one root brick and as its eight
children of half the size gives the same cells, and the same CFL step, in
every reconstruction and precision."""

import numpy as np
import pytest

from test_brick_shapes_gpu import state


@pytest.mark.gpu
@pytest.mark.parametrize("half", [8, 12, 20])
@pytest.mark.parametrize("bw,recon", [(2, 0), (3, 1), (4, 1)])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_large_root_brick_equals_its_children(gpu, half, bw, recon, prec):
    n = 2 * half
    u = state(n)
    cfg = dict(physics=gpu.PHYSICS_EULER, grid_dim=0.5, z_reflect=0, max_bricks=9, bw=bw, reconstruction=recon,
               precision=gpu.PREC_MIXED if prec == "mixed" else gpu.PREC_FP64)
    inner = (slice(bw, -bw),) * 3
    a = gpu.AMR(nx=n, max_refine_level=1, **cfg)
    a.init()
    U = np.zeros((1, 6) + (n + 2 * bw,) * 3)
    U[(0, slice(None)) + inner] = u
    a.upload_state(U)
    a.enforce_boundaries()
    b = gpu.AMR(nx=half, max_refine_level=1, **cfg)
    loc = [(c & 1, (c >> 1) & 1, c >> 2) for c in range(8)]
    part = [(slice(None),) + tuple(slice(q * half, (q + 1) * half) for q in reversed(l)) for l in loc]
    b.load_tree([0] + [1] * 8, [(0, 0, 0)] + loc)
    V = np.zeros((9, 6) + (half + 2 * bw,) * 3)
    for c in range(8):
        V[(1 + c, slice(None)) + inner] = u[part[c]]
    b.upload_state(V)
    b.inject_from_children()
    b.enforce_boundaries()
    dt = a.max_dt()
    # the coarse root allows a longer step; the tree's reciprocals cost a few roundings
    np.testing.assert_allclose(b.max_dt(), dt, rtol=16e-16)
    for x in (a, b):
        x.store()
        for beta in (1.0, 0.25, 2.0 / 3.0):
            x.sub_step(dt, beta)
            x.inject_from_children()
    got, want = b.download_state(), a.download_state()[(0, slice(None)) + inner]
    # the FP32 flux may be contracted differently for another brick size: a
    # few of its roundings (2^-24) in each of three substeps
    tol = np.abs(want).max(axis=(1, 2, 3)) * (64 * 2.0 ** -24 if prec == "mixed" else 0.0)
    for c in range(8):
        err = np.abs(got[(1 + c, slice(None)) + inner] - want[part[c]]).max(axis=(1, 2, 3))
        assert np.all(err <= tol), (c, err)
    a.close()
    b.close()
