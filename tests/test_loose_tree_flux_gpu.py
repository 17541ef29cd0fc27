"""Coarse-fine flux corrections on loaded trees that are not properly nested:
a corrected face can then be read by two coarse bricks, the parent and the
parent's neighbour, and both have to be corrected.  Ghosts and a substep
against the restatement of the reference's operations."""

import numpy as np
import pytest

import amr_oracle as oracle
from test_small_brick_ghosts_gpu import check_against_oracle


def double_readers(T):
    """Corrections of a brick other than the child's parent that read a face
    corrected itself."""
    count = 0
    for i in range(1, T.n):
        p = T.parent[i]
        for f in range(6):
            ax, side = f >> 1, f & 1
            if T.is_phys(i, f) or T.neighbor(i, f) is not None:
                continue
            if not any(T.child[i, c] >= 0 for c in range(8) if (c >> ax) & 1 == side):
                continue
            if (T.cidx[i] >> ax) & 1 == side and T.neighbor(p, f) is not None:
                count += 1
    return count


def random_tree(seed, n, levels):
    rng = np.random.default_rng(seed)
    nodes = {(0, 0, 0, 0)}
    while len(nodes) < n:
        l, x, y, z = sorted(nodes)[rng.integers(len(nodes))]
        if l < levels:
            c = rng.integers(0, 2, 3)
            nodes.add((l + 1, int(2 * x + c[0]), int(2 * y + c[1]), int(2 * z + c[2])))
    order = []

    def walk(l, x, y, z):
        order.append((l, x, y, z))
        for c in range(8):
            ch = (l + 1, 2 * x + (c & 1), 2 * y + ((c >> 1) & 1), 2 * z + (c >> 2))
            if ch in nodes:
                walk(*ch)

    walk(0, 0, 0, 0)
    a = np.array(order)
    return a[:, 0], a[:, 1:]


@pytest.mark.gpu
@pytest.mark.parametrize("nx,bw,recon", [(8, 2, 0), (8, 3, 1)])
def test_smallest_tree_with_two_readers(gpu, nx, bw, recon):
    level = [0, 1, 2, 3, 1]
    loc = [(0, 0, 0), (0, 0, 0), (1, 0, 0), (3, 0, 0), (1, 0, 0)]
    T = check_against_oracle(gpu, level, loc, nx, bw, recon)
    assert double_readers(T) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("seed,n,levels", [(1, 30, 4), (2, 60, 4), (3, 60, 5), (4, 12, 2)])
@pytest.mark.parametrize("nx,bw,recon", [(4, 2, 0), (4, 4, 1), (8, 2, 0)])
def test_random_trees(gpu, seed, n, levels, nx, bw, recon):
    level, loc = random_tree(seed, n, levels)
    check_against_oracle(gpu, level, loc, nx, bw, recon)
    if levels > 2:
        assert double_readers(oracle.Tree(level, loc, bw=bw, nx=nx)) > 0
