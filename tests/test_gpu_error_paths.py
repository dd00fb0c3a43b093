"""GPU: calls on a handle after one of its calls failed on the host."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

SPEC = O.henon_spec()
# launches of more points than the warps' first pieces (the rest comes from the work queue)
N, DEPTH = 60001, 18


def boxes(seed):
    codes = np.random.default_rng(seed).choice(2 ** DEPTH, size=N, replace=False)
    return np.sort(codes).astype(np.uint64), np.full(N, DEPTH, np.uint8), np.zeros(N, np.uint8)


@pytest.mark.parametrize("stage", [1, 2])
@pytest.mark.parametrize("launches,steps", [(1, 2), (2, 3), (3, 1)])
def test_searches_after_a_run_whose_graph_failed(stage, launches, steps):
    """A fused run whose graph cannot be made or launched leaves the work queue's counters to
    the launches that ran: the next launch images every point."""
    import b12_b200 as B
    from b12_b200 import _lib
    sc = B.Scheme(B.henon(), B.inner_grid(4))
    t = B.ImplicitBoxTree(SPEC["center"], SPEC["radius"])
    t.load_leaves(*boxes(0))
    for _ in range(launches):
        t.search_by_image(sc)
    assert _lib.lib().b12g_tree_refuse_graph(t._h, stage) == 0
    with pytest.raises(B.B12gError) as e:
        t.subdivision_run(sc, steps)
    assert e.value.status == _lib.ERR_OOM
    o = O.Oracle(SPEC)
    for seed in (1, 2):                  # (other leaves than the ones searched before)
        t.load_leaves(*boxes(seed))
        o.load(*boxes(seed))
        assert np.array_equal(t.search_by_image(sc), o.search_by_image())
    want, _ = o.subdivision(steps)       # the request held for one run
    assert list(t.subdivision_run(sc, steps)) == list(want)
    assert np.array_equal(t.search_by_image(sc), o.search_by_image())
    t.close()
