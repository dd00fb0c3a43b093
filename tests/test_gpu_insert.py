"""GPU: insertion of points at one depth (the boxes sorted by their codes alone) against the
oracle: code lengths at the sort's digits, repeated points, depths below and inside the tree."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SPEC = O.coupled_duffing_spec(8, 0)


@pytest.mark.parametrize("depth", [1, 7, 8, 9, 16, 17, 24, 33, 56, 57, 64])
@pytest.mark.parametrize("n", [1, 2, 37, 4095, 4097])
def test_points_into_boxes_of_another_depth(depth, n):
    import b12_b200 as B
    rng = np.random.default_rng([depth, n])
    pts = rng.normal(size=(n, 4)) * 0.9          # some outside the domain
    pts[n // 2:] = pts[: n - n // 2]             # every box at least twice where there is room
    for first, hit in ((0, B.NONE), (3, B.HIT)):     # into the surrounding box; into boxes of depth 3
        t = B.ImplicitBoxTree(SPEC["center"], SPEC["radius"])
        o = O.Oracle(SPEC)
        if first:
            seeds = rng.uniform(-1.9, 1.9, size=(9, 4))
            t.insert_points(seeds, first)
            o.insert_points_general(seeds, first)
        got, want = t.insert_points(pts, depth, B.INS, hit), o.insert_points_general(pts, depth, 2, int(hit))
        assert got == (want[0] if isinstance(want, tuple) else want)
        for x, y in zip(t.leaves(), o.leaves()):
            assert np.array_equal(x, y)
        t.close()
