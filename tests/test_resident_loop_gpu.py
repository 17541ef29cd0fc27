"""The shared-memory relaxation loop of the persistent solve where it can go
wrong: levels of one brick (decided by its own block), of as many bricks as
blocks (the block that forms the sums holds one too), and of more (up to
four bricks in a block), on 8^3 and 12^3 bricks, in every block layout.  Every
layout, and the plain solve (one launch, or the host's loop over launches
where it is profiled), must give the same potential bit for bit in FP64 and in
the mixed form; relaxation passes are counted alike."""

import importlib.util
import os

import numpy as np
import pytest

from conftest import PKG, _load_pkg_module

spec = importlib.util.spec_from_file_location("amr_initial", os.path.join(PKG, "initial.py"))
initial = importlib.util.module_from_spec(spec)
spec.loader.exec_module(initial)

PREC = {"fp64": 0, "mixed": 1}


def star(gpu, prec, persistent):
    a = gpu.AMR(physics=gpu.PHYSICS_EULER_GRAVITY, max_refine_level=4, grid_dim=0.5, z_reflect=0, max_bricks=1024,
                precision=prec, persistent_solve=persistent)
    initial.build_tree(a, "polytrope", 1.0e-6, 0.5, 0, 4, device=True, ghosts=False)
    return a, 1.0e-5


def binary(gpu, prec, persistent, helm):
    P = initial.binary_params()
    a = gpu.AMR(physics=gpu.PHYSICS_ZTWD, nf=13, bw=3, nx=12, reconstruction=gpu.RECON_PPM, grid_dim=1.0, z_reflect=1,
                mirror_refine_y=1, max_refine_level=5, rho_floor=initial.BINARY["rho_floor"], max_bricks=512,
                precision=prec, persistent_solve=persistent)
    a.ztwd_set_eos(helm)
    a.ztwd_set_frame(P["omega"], P["omega"], 0.0, 0.0)
    a.init()
    U = initial.evaluate("binary", a.get_tree(), 3, 12, 1.0, 1, 5, ghosts=False)
    initial.build_tree(a, "binary", float(U[:, 0].max()) / 1.0e6, 1.0, 1, 5, device=True, ghosts=False)
    return a, 1.0e-4


@pytest.mark.gpu
@pytest.mark.parametrize("nx,layouts", [(8, ((0, 1), (0, 2), (1, 1), (1, 2), (1, 0))),
                                        (12, ((1, 1), (0, 1), (0, 2), (2, 1), (2, 0)))])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_layouts_give_the_same_bits(gpu, table_path, nx, layouts, prec):
    """8^3: levels of 1, 8, 64, 160 and 408 bricks on 148 blocks and up
    (three bricks a block, then two, then one).  12^3: levels of 1, 8, 32,
    48, 72 and 148 bricks (as many as the blocks of one per SM)."""
    helm = None
    if nx == 12:
        P = initial.binary_params()
        helm = _load_pkg_module("helm_b200", "helm.py").Helm(table_path)
        helm.set_cgs_units(P["cm"], P["g"], P["s"], 1.0)

    def solve(persistent, layout=None, host_loop=True):
        a, tol = star(gpu, PREC[prec], persistent) if nx == 8 else binary(gpu, PREC[prec], persistent, helm)
        if layout is not None:
            a.set_solve_layout(*layout)
            e, n = a.graph_solve(tol)
        else:
            a.profile(host_loop)  # a profiled solve runs the host's loop, launch by launch
            e, n = a.poisson_solve(tol)
        out = e, n, a.relax_passes(), a.download_poisson()
        a.close()
        return out

    want = solve(0)
    got = solve(0, host_loop=False)  # the plain solve's one launch
    assert got[:2] == want[:2] and all(np.array_equal(x, y) for x, y in zip(got[2:], want[2:]))
    for layout in layouts:
        got = solve(4, layout)
        assert got[0] == want[0] and got[1] == want[1], layout
        assert np.array_equal(got[2], want[2]), layout
        assert np.array_equal(got[3], want[3]), layout
    if helm is not None:
        helm.close()


@pytest.mark.gpu
def test_plain_solve_limits(gpu):
    """The plain solve's one launch keeps the host loop's answers at its
    limits: the V-cycle cap (also 0), and waits too short for the launch,
    after which the host's loop gives the same potential."""
    a, tol = star(gpu, 0, 0)
    with pytest.raises(gpu.AmrError) as e:
        a.poisson_solve(tol, 0)
    assert e.value.code == -4
    with pytest.raises(gpu.AmrError) as e:
        a.poisson_solve(tol, 2)
    assert e.value.code == -4
    b, _ = star(gpu, 0, 0)
    b.profile(True)
    with pytest.raises(gpu.AmrError) as e:
        b.poisson_solve(tol, 2)
    assert e.value.code == -4
    assert np.array_equal(a.download_poisson(), b.download_poisson())
    a.set_wait_limit(1)
    assert a.poisson_solve(tol) == b.poisson_solve(tol)
    assert np.array_equal(a.download_poisson(), b.download_poisson())
    a.set_wait_limit(0)
    a.close()
    b.close()
