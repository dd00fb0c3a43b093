"""GPU: a saved matrix whose first values are counts over fewer points than the others."""
import numpy as np
import pytest

from test_gpu_measure import matrix, near

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,spread,halves", [(130000, 400, 2000), (130000, 400, 129999), (1000, 7, 600)])
def test_the_loaded_matrix_gives_the_same_bits(n, spread, halves, tmp_path):
    """(130,000 boxes: more entries than stay on chip in FP64, 1,000: fewer)"""
    import b12_b200 as B
    rng = np.random.default_rng([n, halves])
    targets = near(np.arange(n), n, rng, 16, spread)
    a = targets[:halves, :1]
    targets[:halves] = np.where(np.arange(16) < 10, a, (a + 1) % n)      # 10/16 and 6/16: counts over 8
    m = matrix(targets, n)
    m.save(tmp_path / "m.json")
    loaded = B.CsrMatrix.load(tmp_path / "m.json")
    assert np.array_equal(loaded.invariant_measure(30), m.invariant_measure(30))
    a, b = loaded.invariant_measure_tol(1e-9, 60, 10), m.invariant_measure_tol(1e-9, 60, 10)
    assert np.array_equal(a[0], b[0]) and a[1:] == b[1:]
