"""GPU: batches and served jobs whose steps are screened in part: past the depth at which the
bound ends, and with instances that it does not cover beside ones that it does."""
import numpy as np
import pytest

from test_screen import forced, lorenz

pytestmark = pytest.mark.gpu

# the forced map's bound ends at depth 26; its steps past that have enough points to be timed
# by the first run's tuning, which the second run replays
FORCED = ([(0.25, -1.0, 1.0, 0.3), (0.25, -1.0, 1.0, 0.05), (0.25, -1.0, 1.0, 0.25), (0.25, -1.0, 1.0, 0.35)],
          [28, 9, 26, 27])
# (10, 900, 8/3) leaves the bound at every depth; the third and fourth batch hold mostly such
COVERED, NOT = (10.0, 28.0, 8.0 / 3.0), (10.0, 900.0, 8.0 / 3.0)
LORENZ = [([COVERED, NOT, COVERED], [13, 13, 9]), ([COVERED, NOT], [12, 12]), ([NOT, COVERED, NOT], [12, 12, 12]),
          ([NOT, COVERED, NOT], [8, 13, 8])]


def compare(spec, maps, params, grid, depths):
    import b12_b200 as B
    from b12_b200.server import JobServer
    b = B.Batch(spec["center"], spec["radius"], B.Scheme(maps[0], grid), params, depths)
    with JobServer() as srv:
        ids = [srv.submit(spec["center"], spec["radius"], m, grid, d) for m, d in zip(maps, depths)]
        srv.wait_all(ids)
        for absolute in (False, True):
            b.run()
            b.transition_matrices(absolute, absolute)
            for k, (m, d) in enumerate(zip(maps, depths)):
                t = B.ImplicitBoxTree(spec["center"], spec["radius"])
                sc = B.Scheme(m, grid)
                counts = t.subdivision_run(sc, d)
                assert np.array_equal(b.counts(k), counts)
                if t.depth() == d:           # (batches and jobs keep no rows of an instance that lost every box)
                    want = t.transition_matrix(sc, absolute, absolute).to_host()
                    for x, y in zip(b.leaves(k), t.leaves()):
                        assert np.array_equal(x, y)
                    for x, y in zip(b.csr(k), want):
                        assert np.array_equal(x, y)
                    if not absolute:
                        r = srv.result(ids[k])
                        for x, y in zip((r["codes"], r["rowptr"], r["cols"], r["vals"]), (t.leaves()[0], *want)):
                            assert np.array_equal(x, y)
                t.close()
    info = b.info()
    b.close()
    return info


def test_forced_batch_past_the_bound():
    import b12_b200 as B
    params, depths = FORCED
    info = compare(forced(), [B.forced_duffing(200, *p) for p in params], params, B.inner_grid(4), depths)
    # the steps past the bound run in a shape of the map's own kernel
    assert info["chunk"] >= 8192


def test_forced_batch_within_the_bound():
    import b12_b200 as B
    params, depths = FORCED[0], [20, 9, 26, 11]
    info = compare(forced(), [B.forced_duffing(200, *p) for p in params], params, B.inner_grid(4), depths)
    assert info["chunk"] < 8192          # every step screened: that kernel's shape


@pytest.mark.parametrize("case", range(len(LORENZ)))
@pytest.mark.parametrize("fma", [False, True])
def test_lorenz_instances_the_bound_does_not_cover(case, fma):
    import b12_b200 as B
    params, depths = LORENZ[case]
    info = compare(lorenz(), [B.lorenz(*p, fma=fma) for p in params], params, B.inner_grid(4), depths)
    assert (info["chunk"] >= 8192) == (case == 2 or case == 3)
