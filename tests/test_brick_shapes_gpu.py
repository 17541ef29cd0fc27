"""The hydro kernels at another brick size and more ghosts than the
reconstruction reads: the same 8^3 grid as one root brick and as its eight
4^3 children gives the same cells bit for bit, and the same CFL step."""

import numpy as np
import pytest


def state(n, seed=5):
    rng = np.random.default_rng(seed)
    x = (np.arange(n) + 0.5) / n - 0.5
    X, Y, Z = x[None, None, :], x[None, :, None], x[:, None, None]
    rho = 1.0 + 0.4 * np.exp(-40.0 * (X * X + Y * Y + Z * Z)) + 0.1 * rng.random((n, n, n))
    v = [0.3 * np.sin(2 * np.pi * (X + 2 * Y)) + 0 * Z, 0.2 + 0.1 * rng.random((n, n, n)), -0.1 + 0 * X + 0 * Y + Z]
    ei = rho ** (5.0 / 3.0) / (2.0 / 3.0)
    ek = 0.5 * rho * sum(w * w for w in v)
    return np.stack([rho] + [rho * w for w in v] + [ei + ek, ei ** 0.6])


@pytest.mark.gpu
@pytest.mark.parametrize("half,bw,recon", [(4, 2, 0), (4, 3, 1), (4, 4, 0), (4, 4, 1)])
def test_root_brick_equals_its_children(gpu, half, bw, recon):
    n = 2 * half
    u = state(n)
    cfg = dict(physics=gpu.PHYSICS_EULER, grid_dim=0.5, z_reflect=0, max_bricks=16, bw=bw, reconstruction=recon)
    a = gpu.AMR(nx=n, max_refine_level=1, **cfg)
    a.init()
    U = np.zeros((1, 6) + (n + 2 * bw,) * 3)
    U[0, :, bw:-bw, bw:-bw, bw:-bw] = u
    a.upload_state(U)
    a.enforce_boundaries()
    b = gpu.AMR(nx=half, max_refine_level=1, **cfg)
    loc = [(c & 1, (c >> 1) & 1, c >> 2) for c in range(8)]
    b.load_tree([0] + [1] * 8, [(0, 0, 0)] + loc)
    V = np.zeros((9, 6) + (half + 2 * bw,) * 3)
    for c, (i, j, k) in enumerate(loc):
        V[1 + c, :, bw:-bw, bw:-bw, bw:-bw] = u[:, k * half:(k + 1) * half, j * half:(j + 1) * half,
                                                i * half:(i + 1) * half]
    b.upload_state(V)
    b.inject_from_children()
    b.enforce_boundaries()
    dt = a.max_dt()
    # the root's coarse cells allow a longer step; nested reciprocals cost a
    # few roundings
    np.testing.assert_allclose(b.max_dt(), dt, rtol=4e-16 * 4)
    for x in (a, b):
        x.store()
        for beta in (1.0, 0.25, 2.0 / 3.0):
            x.sub_step(dt, beta)
            x.inject_from_children()
    got, want = b.download_state(), a.download_state()[0, :, bw:-bw, bw:-bw, bw:-bw]
    for c, (i, j, k) in enumerate(loc):
        assert np.array_equal(got[1 + c, :, bw:-bw, bw:-bw, bw:-bw],
                              want[:, k * half:(k + 1) * half, j * half:(j + 1) * half, i * half:(i + 1) * half]), c
    # the restricted root: means of eight cells, in the reference's order
    s = np.zeros((6, half, half, half))
    for dk in (0, 1):
        for dj in (0, 1):
            for di in (0, 1):
                s = s + want[:, dk::2, dj::2, di::2]
    root = got[0, :5, bw:-bw, bw:-bw, bw:-bw]
    assert np.array_equal(root, (s * 0.125)[:5])
    a.close()
    b.close()
