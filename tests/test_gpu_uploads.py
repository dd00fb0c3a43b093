"""GPU: calls that read uploaded inputs right after the call that uploaded them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_largest_batch_runs_right_after_its_creation():
    import b12_b200 as B
    n, grid = 512, B.inner_grid(2)
    center, radius = (0.0, 0.0, 27.0), (30.0, 30.0, 40.0)
    rho = 20.0 + 15.0 * np.arange(n) / n
    depths = [18 - 3 * (i % 5) for i in range(n)]
    for _ in range(3):
        b = B.Batch(center, radius, B.Scheme(B.lorenz(), grid), [(10.0, r, 8.0 / 3.0) for r in rho], depths)
        b.run()
        for i in (0, 5, 255, 494, 510, 511):
            t = B.ImplicitBoxTree(center, radius)
            assert np.array_equal(b.counts(i), t.subdivision_run(B.Scheme(B.lorenz(rho=rho[i]), grid), depths[i]))
            for x, y in zip(b.leaves(i), t.leaves()):
                assert np.array_equal(x, y)
            t.close()
        b.close()


def test_loaded_matrix_is_read_right_after_its_upload(tmp_path):
    import b12_b200 as B
    from b12_b200.tree import json_write_coo
    n = 60000
    rng = np.random.default_rng(2)
    cols = np.sort(rng.integers(0, n, size=(n, 5)), axis=1).astype(np.uint32)
    keep = np.concatenate([np.ones((n, 1), bool), cols[:, 1:] != cols[:, :-1]], axis=1)
    rowptr = np.concatenate([[0], np.cumsum(keep.sum(axis=1))]).astype(np.uint32)
    cols, vals = cols[keep], rng.uniform(0.1, 1.0, size=int(rowptr[-1]))
    json_write_coo(tmp_path / "m.json", n, n, rowptr, cols, vals)
    got = B.CsrMatrix.load(tmp_path / "m.json").to_host()
    for x, y in zip(got, (rowptr, cols, vals)):
        assert np.array_equal(x, y)
