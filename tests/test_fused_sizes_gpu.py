"""The fused substep is written for bricks of 8^3 with two ghost layers; any
other shape is refused before a launch and leaves the state as it was."""

import numpy as np
import pytest

import amr_oracle as oracle
from test_small_brick_ghosts_gpu import random_state


@pytest.mark.gpu
@pytest.mark.parametrize("nx,bw,recon", [(4, 2, 0), (12, 2, 0), (16, 2, 0), (8, 3, 0), (8, 3, 1)])
def test_other_bricks_are_refused(gpu, nx, bw, recon):
    T = oracle.Tree([0], [(0, 0, 0)], bw=bw, nx=nx)
    a = gpu.AMR(physics=gpu.PHYSICS_EULER, nx=nx, bw=bw, reconstruction=recon, max_bricks=1, grid_dim=0.5, z_reflect=0,
                max_refine_level=0)
    a.load_tree(T.level, T.loc)
    a.upload_state(random_state(1, T.gnx, bw, 3))
    U = a.download_state()
    a.store()
    with pytest.raises(gpu.AmrError) as e:
        a.fused_sub_step(1.0e-3, 1.0)
    assert e.value.code == -1
    assert np.array_equal(a.download_state(), U)
    a.close()
