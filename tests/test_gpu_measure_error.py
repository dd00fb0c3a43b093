"""GPU: the power iteration's rounding error on matrices too large for its FP64 entries to stay
on chip (packed entries, rows summed in pairs), against the same iteration in 80 bits."""
import numpy as np
import pytest

from test_gpu_measure import matrix, near

pytestmark = pytest.mark.gpu


def measure_in_80_bits(n, rowptr, cols, vals, iters):
    order = np.argsort(cols, kind="stable")
    src = np.repeat(np.arange(n, dtype=np.int64), np.diff(rowptr))[order]
    w, c = vals[order].astype(np.longdouble), cols[order]
    heads = np.flatnonzero(np.concatenate([[True], c[1:] != c[:-1]]))
    v = np.full(n, np.longdouble(1.0) / np.longdouble(n))
    for _ in range(iters):
        sums = np.add.reduceat(w * v[src], heads)
        v = np.zeros(n, np.longdouble)
        v[c[heads]] = sums
        v /= v.sum()
    return v


# A row's sum in a pair is rounded once (at most u = 2^-53, 0.41 u in the mean square) and its
# product with 1 / norm once more; the norm's own roundings shift all entries alike by less than
# u / 2 in the mean square; a row averages the earlier iterates' errors over its ten sources and
# more (0.2 u).  Together 0.8 u: 0.9e-16.  (One sum from start to end gives 1.3 to 2.0e-16.)
@pytest.mark.parametrize("n,P,spread,iters,seed", [(300000, 16, 40, 40, 1), (300000, 16, 9, 25, 2),
                                                   (260000, 16, 60, 24, 3), (600000, 16, 40, 17, 4),
                                                   (265000, 32, 120, 20, 5)])
def test_measure_of_a_large_matrix(n, P, spread, iters, seed):
    m = matrix(near(np.arange(n), n, np.random.default_rng(seed), P, spread), n)
    rowptr, cols, vals = m.to_host()
    if spread > 9:
        assert m.nnz > 13312 * 148       # 13 FP64 entries a thread: the smaller kernel's room
    want = measure_in_80_bits(n, rowptr, cols, vals, iters)
    got = m.invariant_measure(iters)
    err = float(np.sqrt((((got - want) ** 2).sum() / (want ** 2).sum())))
    print(f"n = {n}, {m.nnz} entries, {iters} iterations: error {err:.3e}")
    assert err < 1.0e-16
    m.close()
