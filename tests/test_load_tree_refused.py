"""A list of bricks that amr_load_tree refuses leaves the context's tree as it
was (host-only contexts: the octree alone)."""

import numpy as np
import pytest

LEVEL = [0, 1, 2, 1]
LOC = [(0, 0, 0), (0, 0, 0), (1, 1, 0), (1, 0, 0)]

BAD = {
    "no root first": ([1, 2], [(0, 0, 0), (0, 0, 0)]),
    "a level left out": ([0, 2], [(0, 0, 0), (0, 0, 0)]),
    "a second root": ([0, 1, 0], [(0, 0, 0), (1, 0, 0), (0, 0, 0)]),
    "a negative level": ([0, 1, -1], [(0, 0, 0), (1, 0, 0), (0, 0, 0)]),
    "not the parent's child": ([0, 1, 2], [(0, 0, 0), (1, 0, 0), (0, 0, 0)]),
    "a negative location": ([0, 1], [(0, 0, 0), (-1, 0, 0)]),
    "listed twice": ([0, 1, 2, 1], [(0, 0, 0), (1, 0, 0), (2, 0, 0), (1, 0, 0)]),
    "twice in a row": ([0, 1, 1], [(0, 0, 0), (1, 0, 0), (1, 0, 0)]),
}


@pytest.mark.parametrize("name", sorted(BAD))
def test_the_tree_stays(amr_mod, name):
    a = amr_mod.AMR(max_bricks=0, max_refine_level=3, grid_dim=0.5, z_reflect=0, mirror_refine_y=0)
    a.load_tree(LEVEL, LOC, np.arange(4))
    before = a.get_tree()
    with pytest.raises(amr_mod.AmrError) as e:
        a.load_tree(*BAD[name])
    assert e.value.code == -1
    after = a.get_tree()
    assert a.nbricks == 4 and np.array_equal(after["level"], LEVEL)
    for k in before:
        assert np.array_equal(before[k], after[k]), k
    # and it still works as a tree
    assert a.refine_from_flags(np.ones((4, 8), np.uint8))
    a.close()


def test_accepted_lists(amr_mod):
    a = amr_mod.AMR(max_bricks=0, max_refine_level=3, grid_dim=0.5, z_reflect=0)
    for level, loc in (([0], [(0, 0, 0)]), (LEVEL, LOC), ([0, 1, 1, 2, 3, 2], [(0, 0, 0), (1, 1, 1), (0, 0, 1), (0, 0, 2),
                                                                              (1, 1, 5), (1, 1, 3)])):
        a.load_tree(level, loc)
        t = a.get_tree()
        # the same bricks (get_tree lists children by octant)
        assert sorted(zip(level, map(tuple, loc))) == sorted(zip(t["level"].tolist(), map(tuple, t["loc"].tolist())))
    a.close()
