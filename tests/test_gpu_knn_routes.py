"""Which kNN calls take the exact path, and what a row order costs the candidate pass."""
import numpy as np
import pytest

from test_gpu_knn import _data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,exact", [(1792, True), (1793, True), (2047, True), (2048, False)])
def test_long_lists_of_small_sets_are_exact(ub, oracle, n, exact):
    """k > 32 and fewer than 2,048 rows: every row recomputed, whatever the number of 256-row tiles."""
    X = _data(n, 12, seed=n)
    gi, gd, rec = ub.knn_bruteforce(X, 100, return_stats=True)
    oi, od = oracle.knn_bruteforce(X, 100)
    assert np.array_equal(gi, oi) and np.array_equal(gd, od)
    assert rec == n if exact else rec < n // 20
