"""Coarse-fine ghosts of 4^3 bricks with three and four ghost layers.  An
octant of such a brick is two cells wide, so the slope of a deep ghost can
read past its parent's other side, where the parent's own ghost may be
coarse-fine as well: every stored face ghost, and a substep, against the
level-ordered restatement of the reference's fill."""

import numpy as np
import pytest

import amr_oracle as oracle
from cases import FP64_FIELD_RTOL, field_rel_err


def ball_tree(amr, nx, bw, levels):
    """The library's own regrid, host only: a ball off the centre, refined."""
    host = amr.AMR(max_bricks=0, nx=nx, bw=bw, max_refine_level=levels, grid_dim=0.5, z_reflect=0,
                   mirror_refine_y=0)
    host.init()
    for _ in range(levels + 1):
        t = host.get_tree()
        flags = np.zeros((len(t["level"]), 8), np.uint8)
        for i, (lv, loc) in enumerate(zip(t["level"], t["loc"])):
            for c in range(8):
                x = (2.0 * loc + np.array([c & 1, (c >> 1) & 1, c >> 2]) + 0.5) / 2.0 ** (lv + 1)
                r = 0.5 * 3.0 ** 0.5 / 2.0 ** (lv + 1)
                flags[i, c] = np.abs(np.linalg.norm(x - [0.3, 0.35, 0.4]) - 0.06) < r
        if not host.refine_from_flags(flags):
            break
    t = host.get_tree()
    host.close()
    return t["level"], t["loc"]


def long_stencils(T):
    """Coarse-fine faces whose slopes read a coarse-fine ghost of the parent."""
    count = 0
    amr_face = lambda i, f: not T.is_phys(i, f) and T.neighbor(i, f) is None
    for i in range(1, T.n):
        for f in range(6):
            if not amr_face(i, f):
                continue
            p, ax = T.parent[i], f >> 1
            first = T.offset[i][ax] - 2 * T.offset[p][ax] + (T.gnx - T.bw if f & 1 else 0)
            lo, hi = first // 2 - 1, (first + T.bw - 1) // 2 + 1
            count += (lo < T.bw and amr_face(p, 2 * ax)) or (hi >= T.gnx - T.bw and amr_face(p, 2 * ax + 1))
    return count


def random_state(n, gnx, bw, seed):
    rng = np.random.default_rng(seed)
    U = np.zeros((n, 6, gnx, gnx, gnx))
    s = (slice(None),) + (slice(bw, gnx - bw),) * 3
    nx = gnx - 2 * bw
    for b in range(n):
        rho = 1.0 + rng.random((nx, nx, nx))
        v = rng.uniform(-0.5, 0.5, (3, nx, nx, nx))
        ei = 1.0 + rng.random((nx, nx, nx))
        U[b][s] = np.stack([rho, rho * v[0], rho * v[1], rho * v[2], ei + 0.5 * rho * (v * v).sum(0), ei ** 0.6])
    return U


def face_ghosts(T, U):
    bw, gnx = T.bw, T.gnx
    return np.stack([np.moveaxis(U[(slice(None),) + oracle._sl(f >> 1, gnx - bw if f & 1 else 0, gnx if f & 1 else bw,
                                                               bw, gnx)], 4 - (f >> 1), -1) for f in range(6)])


def check_against_oracle(gpu, level, loc, nx, bw, recon, **cfg):
    T = oracle.Tree(level, loc, bw=bw, nx=nx, grid_dim=0.5)
    a = gpu.AMR(physics=gpu.PHYSICS_EULER, nx=nx, bw=bw, reconstruction=recon, max_bricks=T.n, grid_dim=0.5,
                z_reflect=0, max_refine_level=max(1, int(max(level))), **cfg)
    a.load_tree(level, loc)
    U = random_state(T.n, T.gnx, bw, T.n)
    a.upload_state(U)
    a.enforce_boundaries()
    want = oracle.enforce_boundaries(T, U.copy())
    got = a.download_state()
    assert np.array_equal(face_ghosts(T, got), face_ghosts(T, want))
    a.store()
    dt = 0.05 * T.h.min()
    a.sub_step(dt, 1.0)
    name = "ppm" if recon == gpu.RECON_PPM else "minmod"
    want = oracle.sub_step(T, U.copy(), U.copy(), dt, 1.0, recon=name)
    s = (slice(None), slice(None)) + (slice(bw, -bw),) * 3
    err = field_rel_err(a.download_state()[s], want[s])
    assert np.all(err <= FP64_FIELD_RTOL), err
    a.close()
    return T


@pytest.mark.gpu
@pytest.mark.parametrize("bw,recon", [(3, 0), (3, 1), (4, 0), (4, 1)])
def test_deep_ghosts_of_4_cell_bricks(gpu, bw, recon):
    level, loc = ball_tree(gpu, 4, bw, 4)
    T = check_against_oracle(gpu, level, loc, 4, bw, recon)
    assert long_stencils(T) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("nx,bw,recon", [(4, 2, 0), (8, 2, 0), (8, 4, 1), (12, 3, 1)])
def test_bricks_without_such_stencils(gpu, nx, bw, recon):
    level, loc = ball_tree(gpu, nx, bw, 3)
    T = check_against_oracle(gpu, level, loc, nx, bw, recon)
    assert long_stencils(T) == 0
