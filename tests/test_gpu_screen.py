"""GPU: the image kernels' screened evaluation and work queue against the oracle, on leaf
sets and launch sizes of every kind (search results, matrices and hits, all exact)."""
import numpy as np
import pytest

from oracle import oracle as O
from test_screen import coupled, forced, lorenz

pytestmark = pytest.mark.gpu


def scheme(spec):
    import b12_b200 as B
    ms, gs = spec["map"], spec["grid"]
    m = B.MapSpec(ms["kind"], steps=ms.get("steps", 1), h=ms.get("h", 0.0), p=tuple(ms.get("p", ())),
                  arith=ms.get("fma", 0))
    g = B.GridSpec(gs["kind"], n=gs.get("n", 1), points=gs.get("points", 1), seed=gs.get("seed", 0),
                   eps=gs.get("eps", 0.0))
    return B.Scheme(m, g)


def trees(spec, codes, depth):
    """A tree and an oracle holding the boxes `codes` of one depth."""
    import b12_b200 as B
    codes = np.unique(np.asarray(codes, dtype=np.uint64))
    dep, flags = np.full(len(codes), depth, np.uint8), np.zeros(len(codes), np.uint8)
    t = B.ImplicitBoxTree(spec["center"], spec["radius"])
    t.load_leaves(codes, dep, flags)
    o = O.Oracle(spec)
    o.load(codes, dep, flags)
    return t, o


def covering(spec, depth, n, seed):
    """Boxes that hold images of one another: the boxes hit from random boxes, twice over."""
    rng = np.random.default_rng(seed)
    o = O.Oracle(spec)
    c, r = np.array(spec["center"]), np.array(spec["radius"])
    x = c + r * rng.uniform(-0.6, 0.6, size=(n, spec["dim"]))
    out = []
    for p in x:
        for _ in range(3):
            code, inside = o.point_code64(p)
            if inside:
                out.append(code >> (64 - depth) if depth else 0)
            p = o.map_apply(p)
    return np.array(out, dtype=np.uint64)


CASES = [
    (lorenz(), [0, 1, 5, 18, 27, 36, 54, 55, 60]),
    (lorenz(fma=1), [3, 22, 30, 57]),
    (dict(lorenz(rho=24.0, steps=7), grid=dict(kind=O.GRID_FULL, n=4, eps=0.1)), [9, 25]),
    (dict(lorenz(h=-0.01, steps=3), grid=dict(kind=O.GRID_PHILOX, points=37, seed=5)), [12, 24]),
    (forced(), [0, 2, 15, 20, 26, 27, 36, 40]),
    (dict(forced(p=(0.1, 0.5, 0.7, 0.2)), grid=dict(kind=O.GRID_FULL, n=5, eps=-0.05)), [17]),
    (coupled(), [0, 4, 16, 24, 29, 40, 60]),
    (dict(coupled(h=-0.03, steps=4), grid=dict(kind=O.GRID_INNER, n=3)), [13, 20]),
]


@pytest.mark.parametrize("case,depth", [(i, d) for i, (_, ds) in enumerate(CASES) for d in ds])
def test_search_matrix_and_hits(case, depth):
    import b12_b200 as B
    spec = CASES[case][0]
    t, o = trees(spec, covering(spec, depth, 150, [case, depth]), depth)
    sc = scheme(spec)
    assert np.array_equal(t.search_by_image(sc), o.search_by_image())
    m = t.transition_matrix(sc, invalid_column=True)
    rp, cols, vals, nc = o.transition_matrix(invalid=True)
    got = m.to_host()
    assert m.n_cols == nc and np.array_equal(got[0], rp) and np.array_equal(got[1], cols)
    assert np.array_equal(got[2], vals)
    assert t.set_flags_by_image(sc, B.HIT) == o.set_flags_by_image(1)
    assert np.array_equal(t.leaves()[2], o.leaves()[2])
    m.close()
    t.close()


@pytest.mark.parametrize("n", [1, 2, 3, 5, 63, 64, 65, 3551, 56830, 56832, 56833, 60001])
def test_work_queue_sizes(n):
    """Launches of less than a unit of 32 points up to those that start with larger pieces
    (888 blocks of 8 warps, 4 units each: 56,832 boxes of 16 points), ragged ones between."""
    spec = O.henon_spec()
    rng = np.random.default_rng(n)
    codes = np.sort(rng.choice(2 ** 18, size=n, replace=False)).astype(np.uint64)
    t, o = trees(spec, codes, 18)
    sc = scheme(spec)
    want = o.search_by_image()
    for _ in range(3):                   # the launches take the two queue counters in turn
        assert np.array_equal(t.search_by_image(sc), want)
    t.close()


@pytest.mark.parametrize("n", [14207, 14208, 14209, 14300, 113663, 113664, 113665, 130000])
def test_work_queue_first_pieces(n):
    """7,104 warps: as many units of 32 points as warps (14,208 boxes of 16 points) need no
    counter, 8 times as many start with larger first pieces."""
    test_work_queue_sizes(n)


def test_queue_turns_through_graphs_and_single_launches():
    """Fused runs (an odd and an even number of launches) between single launches."""
    spec = O.henon_spec()
    import b12_b200 as B
    t = B.ImplicitBoxTree(spec["center"], spec["radius"])
    sc = scheme(spec)
    for steps in (7, 8, 7, 1, 8):
        t.delete_depth(0)
        o = O.Oracle(spec)
        want, _ = o.subdivision(steps)
        assert list(t.subdivision_run(sc, steps)) == list(want)
        assert np.array_equal(t.search_by_image(sc), o.search_by_image())
        assert t.set_flags_by_image(sc, B.HIT) == o.set_flags_by_image(1)
    t.close()


LORENZ_BATCHES = [
    # one set of coefficients but rho: screened; strict and FMA, deep and shallow
    ([(10.0, 28.0, 8.0 / 3.0), (10.0, 15.5, 8.0 / 3.0), (10.0, 34.9, 8.0 / 3.0)], [17, 3, 12], 0),
    ([(10.0, 28.0, 8.0 / 3.0), (10.0, 21.0, 8.0 / 3.0)], [1, 16], 1),
    # other sigma and beta too: each map's own arithmetic
    ([(10.0, 28.0, 8.0 / 3.0), (9.5, 28.0, 8.0 / 3.0), (10.0, 28.0, 2.5)], [14, 15, 9], 1),
    # an instance the bound does not cover beside one it does
    ([(10.0, 28.0, 8.0 / 3.0), (10.0, 900.0, 8.0 / 3.0)], [12, 12], 0),
]
FORCED_BATCHES = [
    ([(0.25, -1.0, 1.0, 0.3), (0.25, -1.0, 1.0, 0.05), (0.25, -1.0, 1.0, 0.42)], [13, 15, 6]),
    ([(0.25, -1.0, 1.0, 0.3), (0.2, -1.0, 1.0, 0.3)], [11, 12]),
    ([(0.25, -1.0, -0.01, 0.3), (0.25, -1.0, -0.01, 0.2)], [9, 10]),
]


@pytest.mark.parametrize("which", [("lorenz", i) for i in range(len(LORENZ_BATCHES))] +
                         [("forced", i) for i in range(len(FORCED_BATCHES))])
def test_batches_and_served_jobs_equal_single_trees(which):
    import b12_b200 as B
    from b12_b200.server import JobServer
    name, i = which
    if name == "lorenz":
        params, depths, fma = LORENZ_BATCHES[i]
        spec, maps = lorenz(), [B.lorenz(*p, fma=bool(fma)) for p in params]
        grid = B.inner_grid(4)
    else:
        params, depths = FORCED_BATCHES[i]
        spec, maps = forced(), [B.forced_duffing(200, *p) for p in params]
        grid = B.inner_grid(3)
    b = B.Batch(spec["center"], spec["radius"], B.Scheme(maps[0], grid), params, depths)
    b.run()
    b.run()
    b.transition_matrices()
    with JobServer() as srv:
        ids = [srv.submit(spec["center"], spec["radius"], m, grid, d) for m, d in zip(maps, depths)]
        srv.wait_all(ids)
        for k, (m, d) in enumerate(zip(maps, depths)):
            t = B.ImplicitBoxTree(spec["center"], spec["radius"])
            sc = B.Scheme(m, grid)
            counts = t.subdivision_run(sc, d)
            codes = t.leaves()[0]
            want = t.transition_matrix(sc).to_host()
            r = srv.result(ids[k])
            assert np.array_equal(b.counts(k), counts) and np.array_equal(r["counts"], counts)
            if t.depth() != d:
                t.close()
                continue           # every box was lost: batches and jobs keep no rows for such an instance
            assert np.array_equal(b.leaves(k)[0], codes) and np.array_equal(r["codes"], codes)
            for x, y in zip(b.csr(k), want):
                assert np.array_equal(x, y)
            for x, y in zip((r["rowptr"], r["cols"], r["vals"]), want):
                assert np.array_equal(x, y)
            t.close()
    b.close()


@pytest.mark.parametrize("name,n,full", [("lorenz", 1, False), ("lorenz", 2, True), ("lorenz", 3, False),
                                         ("lorenz", 5, False), ("forced", 6, False), ("forced", 11, True)])
def test_batch_matrices_keep_lost_points(name, n, full):
    """Rows of 1 to 125 points, counts or shares, with the lost column, against the oracle."""
    import b12_b200 as B
    depths = [11, 4, 8]
    if name == "lorenz":
        params = [(10.0, r, 8.0 / 3.0) for r in (28.0, 33.0, 24.5)]
        specs, maps = [lorenz(rho=p[1], fma=1) for p in params], [B.lorenz(*p, fma=True) for p in params]
    else:
        params = [(0.25, -1.0, 1.0, g) for g in (0.3, 0.1, 0.4)]
        specs, maps = [forced(p=p) for p in params], [B.forced_duffing(200, *p) for p in params]
    grid = B.full_grid(n, 0.1) if full else B.inner_grid(n)
    spec_grid = dict(kind=O.GRID_FULL if full else O.GRID_INNER, n=n, eps=0.1 if full else 0.0)
    b = B.Batch(specs[0]["center"], specs[0]["radius"], B.Scheme(maps[0], grid), params, depths)
    b.run()
    for absolute in (False, True):
        b.transition_matrices(absolute, True)
        for i, d in enumerate(depths):
            o = O.Oracle(dict(specs[i], grid=spec_grid))
            want, _ = o.subdivision(d)
            assert list(b.counts(i)) == list(want)
            if want.min() == 0 or o.n == 1:
                continue               # every box was lost: no rows are kept
            for x, y in zip(b.csr(i), o.transition_matrix(absolute, True)):
                assert np.array_equal(x, y)
    b.close()


@pytest.mark.parametrize("case,depth", [(0, 4), (0, 24), (0, 50), (1, 21), (2, 17), (3, 20), (4, 13), (4, 25), (5, 16),
                                        (6, 23), (6, 60), (7, 18)])
def test_leaves_of_several_depths(case, depth):
    """A covering with a third of its boxes split once and a third twice."""
    import b12_b200 as B
    spec = CASES[case][0]
    rng = np.random.default_rng([case, depth, 9])
    base = np.unique(covering(spec, depth, 150, [case, depth]))
    cut = rng.integers(0, 3, size=len(base))
    leaves = []
    for code, c in zip(base, cut):
        for low in range(1 << int(c)):
            if c == 0 or rng.random() < 0.7:
                leaves.append(((int(code) << int(c)) | low, depth + int(c)))
    codes = np.array([x[0] for x in leaves], dtype=np.uint64)
    deps = np.array([x[1] for x in leaves], dtype=np.uint8)
    flags = np.where(rng.random(len(codes)) < 0.5, 8, 0).astype(np.uint8)
    t = B.ImplicitBoxTree(spec["center"], spec["radius"])
    t.load_leaves(codes, deps, flags)
    o = O.Oracle(spec)
    o.load(codes, deps, flags)
    sc = scheme(spec)
    assert np.array_equal(t.search_by_image(sc), o.search_by_image())
    some = B.Scheme(sc.map, sc.grid, flags_to_check=8)
    assert np.array_equal(t.search_by_image(some), o.search_by_image(np.nonzero(flags & 8)[0]))
    m = t.transition_matrix(sc, invalid_column=True)
    rp, cols, vals, nc = o.transition_matrix(invalid=True)
    got = m.to_host()
    assert m.n_cols == nc and np.array_equal(got[0], rp) and np.array_equal(got[1], cols)
    assert np.array_equal(got[2], vals)
    for _ in range(2):
        assert t.set_flags_by_image(sc, B.HIT) == o.set_flags_by_image(1)
    assert np.array_equal(t.leaves()[2], o.leaves()[2])
    m.close()
    t.close()
