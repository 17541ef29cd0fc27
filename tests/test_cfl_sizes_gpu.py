"""The CFL step of every brick size whose pencils one block stages, against
the restatement of the reference's: a two-level tree, both reconstructions
and precisions (the step is formed in FP64 in either)."""

import numpy as np
import pytest

import amr_oracle as oracle
from test_small_brick_ghosts_gpu import random_state


@pytest.mark.gpu
@pytest.mark.parametrize("nx", [4, 8, 12])
@pytest.mark.parametrize("bw,recon", [(2, 0), (3, 0), (3, 1), (4, 1)])
@pytest.mark.parametrize("prec", [0, 1])
def test_max_dt(gpu, nx, bw, recon, prec):
    level, loc = [0, 1, 1, 1], [(0, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 1)]
    T = oracle.Tree(level, loc, bw=bw, nx=nx, grid_dim=0.5)
    a = gpu.AMR(physics=gpu.PHYSICS_EULER, nx=nx, bw=bw, reconstruction=recon, max_bricks=T.n, grid_dim=0.5,
                z_reflect=0, max_refine_level=1, precision=prec)
    a.load_tree(level, loc)
    U = random_state(T.n, T.gnx, bw, 100 * nx + bw)
    a.upload_state(U)
    a.enforce_boundaries()
    U = oracle.enforce_boundaries(T, U)
    want = oracle.max_dt(T, U, 1.3, 5.0 / 3.0, a.cfg.cfl, "ppm" if recon == gpu.RECON_PPM else "minmod")
    # square roots and pow of the pressure differ in the last place
    np.testing.assert_allclose(a.max_dt(), want, rtol=1e-14)
    a.close()
