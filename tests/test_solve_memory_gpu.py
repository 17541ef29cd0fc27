"""The plain solve where the device has no room for the buffers of its one
launch: the host's loop gives the result, nothing of the failed attempt stays
allocated or half made, and once there is room the solve and the graph form
give the same potential."""

import contextlib
import importlib.util
import os

import numpy as np
import pytest
import torch

from conftest import PKG

spec = importlib.util.spec_from_file_location("amr_initial", os.path.join(PKG, "initial.py"))
initial = importlib.util.module_from_spec(spec)
spec.loader.exec_module(initial)

TOL = 1.0e-5
MB = 1 << 20


def star(gpu):
    # a pool large enough for the solve's buffers to be 100 MB (face
    # snapshots), 39 MB (nested sums), 201 MB (tagged snapshots), 131 MB (phi)
    a = gpu.AMR(physics=gpu.PHYSICS_EULER_GRAVITY, max_refine_level=2, grid_dim=0.5, z_reflect=0, max_bricks=16384)
    initial.build_tree(a, "polytrope", 1.0e-6, 0.5, 0, 2, device=True, ghosts=False)
    a.download_poisson()  # the copies' staging buffer, before memory gets short
    a.synchronize()
    return a


@contextlib.contextmanager
def only(leave):
    """All but `leave` bytes of the device's memory taken; the bytes left."""
    torch.cuda.empty_cache()
    p = torch.cuda.caching_allocator_alloc(torch.cuda.mem_get_info()[0] - leave)
    try:
        yield torch.cuda.mem_get_info()[0]
    finally:
        torch.cuda.caching_allocator_delete(p)
        torch.cuda.empty_cache()


def launches(a, call):
    n = a.launch_count()
    call()
    return a.launch_count() - n


@pytest.mark.gpu
@pytest.mark.parametrize("leave", [64 * MB, 170 * MB, 400 * MB])
def test_no_room_for_the_solve(gpu, leave):
    ref = star(gpu)
    P0 = ref.download_poisson()
    ref.profile(True)  # the host's loop; its kernels are loaded with it
    want = ref.poisson_solve(TOL)
    phi = ref.download_poisson()
    ref.close()

    a = star(gpu)
    with only(leave) as free:
        assert launches(a, lambda: a.poisson_solve(TOL)) > 100  # the host's loop
        assert np.array_equal(a.download_poisson(), phi)
        assert free - torch.cuda.mem_get_info()[0] < 32 * MB
        # the graph form fails as a call, and leaves nothing either
        if leave < 100 * MB:
            with pytest.raises(gpu.AmrError) as e:
                a.graph_solve(TOL)
            assert e.value.code == -2
            assert free - torch.cuda.mem_get_info()[0] < 32 * MB
        # no new attempt on the same tree, and the same answer
        a.upload_poisson(P0)
        assert a.poisson_solve(TOL) == want
        assert np.array_equal(a.download_poisson(), phi)
    a.upload_poisson(P0)
    assert a.poisson_solve(TOL) == want
    assert np.array_equal(a.download_poisson(), phi)
    a.upload_poisson(P0)
    assert a.graph_solve(TOL) == want
    assert np.array_equal(a.download_poisson(), phi)
    # a tree loaded again is a new topology: the one launch is back
    t = a.get_tree()
    U = a.download_state()
    a.load_tree(t["level"], t["loc"], t["age"])
    a.upload_state(U)
    a.upload_poisson(P0)
    assert launches(a, lambda: a.poisson_solve(TOL)) < 100
    assert np.array_equal(a.download_poisson()[0], phi[0])
    a.close()
