"""GPU: screened launches at the sizes where their work queues change (592 blocks of 8 warps,
units of 32 points), and matrices refilled by trees on other streams."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_screen import scheme, trees
from test_screen import lorenz

pytestmark = pytest.mark.gpu

SPEC = dict(lorenz(), grid=dict(kind=O.GRID_INNER, n=4))       # 64 points a box: two units


@pytest.mark.parametrize("n", [2367, 2368, 2369, 18943, 18944, 18945, 20011])
def test_leaves_of_one_depth(n):
    """2,368 boxes: a unit for every warp; 18,944: first pieces of four units, and as many left."""
    rng = np.random.default_rng(n)
    codes = np.sort(rng.choice(2 ** 18, size=n, replace=False)).astype(np.uint64)
    t, o = trees(SPEC, codes, 18)
    sc = scheme(SPEC)
    want = o.search_by_image()
    for _ in range(2):
        assert np.array_equal(t.search_by_image(sc), want)
    t.close()


@pytest.mark.parametrize("n", [9471, 9472, 9473, 9475, 12001])
def test_leaves_of_two_depths(n):
    """From 18,944 units on the mixed kernel's warps take four at a time."""
    import b12_b200 as B
    rng = np.random.default_rng(n)
    codes = np.sort(rng.choice(2 ** 17, size=n, replace=False)).astype(np.uint64)
    deps = np.full(n, 17, np.uint8)
    deps[n // 3:] = 18
    codes[n // 3:] = 2 * codes[n // 3:] + 1
    t, o = B.ImplicitBoxTree(SPEC["center"], SPEC["radius"]), O.Oracle(SPEC)
    flags = np.zeros(n, np.uint8)
    t.load_leaves(codes, deps, flags)
    o.load(codes, deps, flags)
    sc = scheme(SPEC)
    want = o.search_by_image()
    assert np.array_equal(t.search_by_image(sc), want)
    assert t.set_flags_by_image(sc, B.HIT) == o.set_flags_by_image(1)
    assert np.array_equal(t.leaves()[2], o.leaves()[2])
    assert np.array_equal(t.search_by_image(sc), want)
    t.close()


def test_matrix_refilled_by_trees_on_other_streams():
    import b12_b200 as B
    a = [B.ImplicitBoxTree(SPEC["center"], SPEC["radius"]) for _ in range(2)]
    sc = scheme(SPEC)
    want = []
    for t, d in zip(a, (21, 20)):
        t.subdivision_run(sc, d)
        want.append(t.transition_matrix(sc, invalid_column=True).to_host())
    m = None
    for k in (0, 1, 0, 0, 1, 1, 0, 1):
        m = a[k].transition_matrix(sc, invalid_column=True, into=m)
        if k == 0:
            continue                     # filled again at once, by this or the other tree
        for x, y in zip(m.to_host(), want[k]):
            assert np.array_equal(x, y)
    m = a[1].transition_matrix(sc, into=m)
    m = a[0].transition_matrix(sc, into=m)
    v = m.invariant_measure(30)
    assert np.array_equal(v, a[0].transition_matrix(sc).invariant_measure(30))
    for t in a:
        t.close()
