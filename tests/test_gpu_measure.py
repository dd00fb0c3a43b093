"""GPU: the power iteration on matrices of counts (packed entries, distinct sources staged in
shared memory) against the oracle, at the edges of its packed form and of its dispatch."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def matrix(targets, n, absolute=False, invalid=False):
    """A matrix from row-major targets (n x P, -1 lost)."""
    import torch
    import b12_b200 as B
    t = B.ImplicitBoxTree([0.0, 0.0], [1.0, 1.0])
    d = max(1, int(np.ceil(np.log2(max(n, 2)))))
    t.load_leaves(np.arange(n, dtype=np.uint64), np.full(n, d, np.uint8), np.zeros(n, np.uint8))
    m = t.transition_rows(torch.from_numpy(targets.astype(np.int32)).cuda(), targets.shape[1], n, absolute, invalid)
    t.close()
    return m


def near(i, n, rng, P, spread):
    """An expanding map with a spread: every row's targets near twice its index."""
    return (2 * i[:, None] + rng.integers(0, spread, size=(len(i), P))) % n


def cases():
    rng = np.random.default_rng(1)
    out = {}
    for n in (1, 2, 31, 32, 33, 1000, 1023, 1025, 20000):
        out[f"near_{n}"] = (near(np.arange(n), n, rng, 5, 7), n)
    # rows of P^T without sources behind one another: up to 127 fit an entry, 128 do not
    for gap in (1, 126, 127, 128, 129, 300):
        n = (gap + 1) * 40
        out[f"gap_{gap}"] = (((near(np.arange(n), 40, rng, 6, 9)) * (gap + 1)) % n, n)
    # counts up to the largest number of points, and one entry a row
    out["one_target"] = (np.repeat(rng.permutation(3000)[:, None], 128, axis=1), 3000)
    out["counts_128"] = (np.sort(rng.integers(0, 3, size=(500, 128)), axis=1) + np.arange(500)[:, None] % 498, 500)
    # rows of P^T with 64 sources (kept on chip) and with 65 (the row-class kernel)
    for k in (64, 65):
        t = np.arange(4000)[:, None].repeat(3, axis=1)
        t[100:100 + k - 1, 0] = 7
        t[7, :] = 7
        out[f"sources_{k}"] = (t, 4000)
    # lost points, and rows that lose every point
    t = near(np.arange(5000), 5000, rng, 8, 11)
    t[rng.random(t.shape) < 0.1] = -1
    t[1234] = -1
    out["lost"] = (t, 5000)
    # scattered sources: a block's distinct sources do not fit beside its entries
    out["scattered"] = (rng.integers(0, 300000, size=(300000, 16)), 300000)
    out["large"] = (near(np.arange(400000), 400000, rng, 12, 24), 400000)
    return out


CASES = cases()


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("absolute", [False, True])
def test_measure_of_counts(name, absolute):
    targets, n = CASES[name]
    if absolute and n > 100000:
        pytest.skip("the large sizes run with relative values")
    m = matrix(targets, n, absolute, invalid=name == "lost")
    rowptr, cols, vals = m.to_host()
    for iters in (0, 1, 2, 9, 30):
        v = m.invariant_measure(iters)
        keep = cols < n
        rows = np.repeat(np.arange(n), np.diff(rowptr))[keep]
        want = np.full(n, 1.0 / n)
        for _ in range(iters):
            want = np.bincount(cols[keep], weights=want[rows] * vals[keep], minlength=n)
            want /= np.abs(want).sum()
        # 64-bit sums of at most 65 products a row, 30 times: far below 1e-12 in L1
        assert np.abs(v - want).sum() < 1e-12
        assert np.array_equal(v, m.invariant_measure(iters))          # the same bits every time
    m.close()


@pytest.mark.parametrize("name", ["near_1000", "gap_127", "gap_128", "counts_128", "lost"])
def test_a_saved_matrix_gives_the_same_bits(name, tmp_path):
    import b12_b200 as B
    targets, n = CASES[name]
    m = matrix(targets, n)
    m.save(tmp_path / "m.json")
    loaded = B.CsrMatrix.load(tmp_path / "m.json")
    assert np.array_equal(loaded.invariant_measure(40), m.invariant_measure(40))
    a, b = loaded.invariant_measure_tol(1e-10, 200, 10), m.invariant_measure_tol(1e-10, 200, 10)
    assert np.array_equal(a[0], b[0]) and a[1:] == b[1:]


def test_weights_that_are_not_counts(tmp_path):
    """A loaded matrix of other values keeps its own arithmetic."""
    import b12_b200 as B
    from b12_b200.tree import json_write_coo
    targets, n = CASES["near_1000"]
    m = matrix(targets, n)
    rowptr, cols, vals = m.to_host()
    w = vals * np.random.default_rng(4).uniform(0.5, 1.5, size=len(vals))
    json_write_coo(tmp_path / "w.json", n, n, rowptr, cols, w)
    v = B.CsrMatrix.load(tmp_path / "w.json").invariant_measure(30)
    assert np.abs(v - O.invariant_measure(rowptr, cols, w, 30)).sum() < 1e-12


def test_refilled_matrix_changes_its_form():
    """A matrix refilled by another tree's rows: the packed form follows."""
    import b12_b200 as B
    sc = B.Scheme(B.henon(), B.inner_grid(4))
    t = B.ImplicitBoxTree([0.0, 0.0], [1.5, 0.45])
    m = None
    for d in (6, 12, 9):
        t.delete_depth(0)
        t.subdivision_run(sc, d)
        m = t.transition_matrix(sc, absolute=d == 9, into=m)
        rowptr, cols, vals = m.to_host()
        assert np.abs(m.invariant_measure(50) - O.invariant_measure(rowptr, cols, vals, 50)).sum() < 1e-12
    t.close()
