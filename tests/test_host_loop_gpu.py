"""The forms that run the multigrid solve in one launch or in a graph, against
the host's loop over launches.  A profiled context runs that loop (it is timed
kernel class by kernel class), so it is the independent side here: the plain
context's own solve is one launch of the same kernel as the persistent form."""

import numpy as np
import pytest

import amr_oracle as oracle
from cases import load_golden
from conftest import _load_pkg_module
from test_graph_gpu import load_state, make
from test_resident_loop_gpu import PREC, binary, initial
from test_small_brick_ghosts_gpu import random_state


def wide_tree():
    """Levels of 1, 8, 64, 512 and 640 bricks."""
    level, loc = [], []
    left = [80]

    def walk(l, x, y, z):
        level.append(l)
        loc.append((x, y, z))
        if l == 3:
            left[0] -= 1
        if l < 3 or (l == 3 and left[0] >= 0):
            for c in range(8):
                walk(l + 1, 2 * x + (c & 1), 2 * y + ((c >> 1) & 1), 2 * z + (c >> 2))

    walk(0, 0, 0, 0)
    return level, loc


@pytest.mark.gpu
@pytest.mark.parametrize("nx,layouts", [(8, ((0, 1), (0, 2), (1, 1))), (12, ((0, 1), (1, 1), (2, 1)))])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_levels_beyond_the_shared_memory_loop(gpu, nx, layouts, prec):
    """Levels of more bricks than the blocks can hold (three or four of 8^3 a
    block, one to four of 12^3; 148 blocks at one per SM) relax through the
    grid barrier, on 8^3 bricks two to a block: three V-cycles' potential and
    passes are the host loop's, bit for bit."""
    level, loc = wide_tree()
    T = oracle.Tree(level, loc, bw=2, nx=nx)
    assert [int((T.level == l).sum()) for l in range(5)] == [1, 8, 64, 512, 640]
    U = random_state(T.n, T.gnx, 2, 5)

    def solve(persistent, layout=None, host_loop=False):
        a = gpu.AMR(physics=gpu.PHYSICS_EULER_GRAVITY, nx=nx, max_refine_level=4, grid_dim=0.5, z_reflect=0,
                    max_bricks=T.n, precision=PREC[prec], persistent_solve=persistent)
        a.load_tree(level, loc)
        a.upload_state(U)
        if layout is not None:
            a.set_solve_layout(*layout)
        a.profile(host_loop)
        with pytest.raises(gpu.AmrError) as e:  # three cycles are not enough
            (a.poisson_solve if layout is None else a.graph_solve)(1.0e-12, 3)
        assert e.value.code == -4
        out = a.relax_passes(), a.download_poisson()[0]
        a.close()
        return out

    want = solve(0, host_loop=True)
    got = solve(0)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
    for layout in layouts:
        got = solve(4, layout)
        assert np.array_equal(got[0], want[0]), layout
        assert np.array_equal(got[1], want[1]), layout


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain", "graph", "persistent"])
def test_star_steps_through_a_regrid(gpu, form):
    """Coupled steps of the two-level star through the regrids at steps 0 and
    8: time steps, trees, state, potential and flow-off of the host's loop."""
    g = load_golden("grav_poly_L2")
    a, b = make(gpu, 2), make(gpu, 2, 1 if form == "persistent" else 0)
    load_state(a, g)
    load_state(b, g)
    a.profile(True)
    last = 0.0
    for s in range(10):
        dt = a.max_dt()
        if s > 0:
            dt = min(1.25 * last, dt)
        last = dt
        a.grav_step(dt, 1.0e-6, 1.0e6, s)
        if form == "plain":
            b.grav_step(dt, 1.0e-6, 1.0e6, s)
        else:
            assert b.graph_grav_step(1.0e-6, 1.0e6, s) == dt
        ta, tb = a.get_tree(), b.get_tree()
        assert np.array_equal(ta["loc"], tb["loc"]) and np.array_equal(ta["age"], tb["age"])
    assert np.array_equal(a.download_state(), b.download_state())
    assert np.array_equal(a.download_poisson()[0], b.download_poisson()[0])
    assert np.array_equal(a.flow_off(), b.flow_off())
    assert np.array_equal(a.relax_passes(), b.relax_passes())
    a.close()
    b.close()


@pytest.mark.gpu
def test_binary_steps_on_the_headline_tree(gpu, table_path):
    """Two BinaryDriver steps of the five-level binary on 12^3 bricks (levels of
    1, 8, 32, 48, 72 and 148): the plain form's one launch and the persistent
    form in four launch shapes give the host loop's state and potential."""
    P = initial.binary_params()
    helm = _load_pkg_module("helm_b200", "helm.py").Helm(table_path)
    helm.set_cgs_units(P["cm"], P["g"], P["s"], 1.0)

    def final(persistent, layout=None, host_loop=False):
        a, tol = binary(gpu, PREC["fp64"], persistent, helm)
        a.enforce_boundaries()
        if layout is not None:
            a.set_solve_layout(*layout)
        a.profile(host_loop)
        dts = []
        for s in range(2):
            dt = a.max_dt()
            if s > 0:
                dt = min(1.25 * dts[-1], dt)
            dts.append(a.ztwd_step(dt, tol, 1.0e6, s))
        b = a.bw
        out = dts, a.download_state()[:, :, b:-b, b:-b, b:-b], a.download_poisson()[0], a.relax_passes()
        a.close()
        return out

    want = final(0, host_loop=True)
    for form in [(0,), (2, (0, 1)), (2, (0, 2)), (2, (1, 1)), (2, (2, 2))]:
        got = final(*form)
        assert got[0] == want[0], form
        assert all(np.array_equal(x, y) for x, y in zip(got[1:], want[1:])), form
    helm.close()
