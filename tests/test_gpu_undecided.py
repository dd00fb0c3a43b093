"""GPU: launches most of whose points the screened evaluation leaves undecided (the warps then
go over to the map's own arithmetic, and back where points are decided again), against the
oracle."""
import numpy as np
import pytest

from oracle import oracle as O
from test_gpu_screen import scheme
from test_screen import forced, lorenz

pytestmark = pytest.mark.gpu

# 2 to 15 % of the points are decided
SPECS = {
    "backward": dict(lorenz(h=-0.02, steps=12, radius=(25.0, 25.0, 25.0)), grid=dict(kind=O.GRID_INNER, n=4)),
    "long_step": dict(lorenz(h=0.02, center=(0.0, 0.0, 0.0), radius=(10.0,) * 3, fma=1),
                      grid=dict(kind=O.GRID_FULL, n=3, eps=0.05)),
    "philox": dict(lorenz(h=-0.02, steps=12, radius=(25.0, 25.0, 25.0), fma=1),
                   grid=dict(kind=O.GRID_PHILOX, points=37, seed=3)),
    "forced": dict(forced(steps=50, p=(-0.25, -1.0, 1.0, 0.3), radius=(1.0, 1.0)), grid=dict(kind=O.GRID_INNER, n=5)),
}


def covering(n, depth, seed):
    """Boxes in runs, so that warps meet many undecided points one after another."""
    rng = np.random.default_rng(seed)
    starts = rng.integers(0, 2 ** depth, size=max(1, n // 50))
    codes = np.unique((starts[:, None] + np.arange(50)[None, :]).ravel() % 2 ** depth)
    return codes.astype(np.uint64)


@pytest.mark.parametrize("name", sorted(SPECS))
@pytest.mark.parametrize("n", [50, 3000, 30000])
def test_leaves_of_one_depth(name, n):
    import b12_b200 as B
    spec, depth = SPECS[name], 18
    codes = covering(n, depth, n)
    dep, flags = np.full(len(codes), depth, np.uint8), np.zeros(len(codes), np.uint8)
    t, o = B.ImplicitBoxTree(spec["center"], spec["radius"]), O.Oracle(spec)
    t.load_leaves(codes, dep, flags)
    o.load(codes, dep, flags)
    sc = scheme(spec)
    assert np.array_equal(t.search_by_image(sc), o.search_by_image())
    m = t.transition_matrix(sc, invalid_column=True)
    rp, cols, vals, nc = o.transition_matrix(invalid=True)
    got = m.to_host()
    assert m.n_cols == nc and np.array_equal(got[0], rp) and np.array_equal(got[1], cols)
    assert np.array_equal(got[2], vals)
    assert t.set_flags_by_image(sc, B.HIT) == o.set_flags_by_image(1)
    assert np.array_equal(t.leaves()[2], o.leaves()[2])
    t.close()


@pytest.mark.parametrize("name", sorted(SPECS))
def test_leaves_of_two_depths(name):
    import b12_b200 as B
    spec, depth = SPECS[name], 17
    codes = covering(20000, depth, 4)
    deep = np.zeros(len(codes), bool)
    deep[::7] = True
    leaves = np.concatenate([np.stack([codes[~deep], np.full((~deep).sum(), depth, np.uint64)], 1),
                             np.stack([codes[deep] * 2 + 1, np.full(deep.sum(), depth + 1, np.uint64)], 1)])
    order = np.argsort(leaves[:, 0] << (np.uint64(depth + 1) - leaves[:, 1]), kind="stable")
    codes, deps = leaves[order, 0].copy(), leaves[order, 1].astype(np.uint8)
    flags = np.zeros(len(codes), np.uint8)
    t, o = B.ImplicitBoxTree(spec["center"], spec["radius"]), O.Oracle(spec)
    t.load_leaves(codes, deps, flags)
    o.load(codes, deps, flags)
    sc = scheme(spec)
    assert np.array_equal(t.search_by_image(sc), o.search_by_image())
    if spec["grid"]["kind"] != O.GRID_PHILOX:
        got = t.transition_matrix(sc, invalid_column=True).to_host()
        for x, y in zip(got, o.transition_matrix(invalid=True)):
            assert np.array_equal(x, y)
    assert t.set_flags_by_image(sc, B.HIT) == o.set_flags_by_image(1)
    t.close()


@pytest.mark.parametrize("name", sorted(SPECS))
def test_continuations_and_insertions(name):
    """From the boxes of 20,000 random points (a continuation's launches, and an insertion's)."""
    import b12_b200 as B
    spec, depth = SPECS[name], 18
    rng = np.random.default_rng(7)
    x0 = np.array(spec["center"]) + np.array(spec["radius"]) * rng.uniform(-1, 1, size=(20000, spec["dim"]))
    t = B.ImplicitBoxTree(spec["center"], spec["radius"])
    counts = t.continuation_run(scheme(spec), x0, depth, max_sweeps=3)
    o, want = O.continuation(spec, depth, x0, max_sweeps=3)
    assert list(counts) == list(want)
    for x, y in zip(t.leaves(), o.leaves()):
        assert np.array_equal(x, y)
    for tree in (t, o):
        tree.set_flags(4)
    sc = scheme(spec)
    sc = B.Scheme(sc.map, sc.grid, depth=depth, flags_to_check=4)
    assert t.insert_by_image(sc, depth, B.INS, B.NONE) == o.insert_by_image(4, 2, 0)
    for x, y in zip(t.leaves(), o.leaves()):
        assert np.array_equal(x, y)
    t.close()


@pytest.mark.parametrize("fma", [False, True])
def test_batches_and_served_jobs(fma):
    import b12_b200 as B
    from b12_b200.server import JobServer
    spec, grid, depths = SPECS["backward"], B.inner_grid(4), [14, 12, 14]
    maps = [B.lorenz(10.0, r, 8.0 / 3.0, h=-0.02, steps=12, fma=fma) for r in (28.0, 24.0, 31.0)]
    b = B.Batch(spec["center"], spec["radius"], B.Scheme(maps[0], grid), [m.p[:3] for m in maps], depths)
    b.run()
    b.transition_matrices()
    with JobServer() as srv:
        ids = [srv.submit(spec["center"], spec["radius"], m, grid, d) for m, d in zip(maps, depths)]
        srv.wait_all(ids)
        for k, (m, d) in enumerate(zip(maps, depths)):
            o = O.Oracle(dict(spec, map=dict(spec["map"], p=list(m.p[:3]), fma=int(fma)),
                              grid=dict(kind=O.GRID_INNER, n=4)))
            want, _ = o.subdivision(d)
            r = srv.result(ids[k])
            assert list(b.counts(k)) == list(want) and list(r["counts"]) == list(want)
            if want.min() == 0 or o.n == 1:
                continue
            assert np.array_equal(b.leaves(k)[0], o.leaves()[0]) and np.array_equal(r["codes"], o.leaves()[0])
            tm = o.transition_matrix()
            for x, y, z in zip(b.csr(k), (r["rowptr"], r["cols"], r["vals"]), tm):
                assert np.array_equal(x, z) and np.array_equal(y, z)
    b.close()
