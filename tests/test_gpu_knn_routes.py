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


@pytest.mark.parametrize("n,classes,k", [(4097, 8, 60), (8000, 16, 100), (16383, 16, 128), (20480, 16, 100)])
def test_alternating_classes(ub, oracle, n, classes, k):
    """Row i in class i % classes, a period that a deal of the caller's order would send to one list: only the few
    rows whose error margin overflows a list are recomputed."""
    g = np.random.Generator(np.random.PCG64(classes))
    X = (g.standard_normal((n, 16)) + 20.0 * g.standard_normal((classes, 16))[np.arange(n) % classes]).astype(np.float32)
    gi, gd, rec = ub.knn_bruteforce(X, k, return_stats=True)
    r1 = min(n, 500)
    oi, od = oracle.knn_bruteforce(X, k, rows=(0, r1))
    assert np.array_equal(gi[:r1], oi) and np.array_equal(gd[:r1], od)
    assert rec < n // 20


@pytest.mark.parametrize("n,d,k", [(10000, 256, 100), (4096, 8, 64)])
def test_ordered_rows(ub, oracle, n, d, k):
    """Points along a line in their order: the 2 S rows next to one another go to as many lists, so none overflows."""
    X = np.repeat(np.arange(n, dtype=np.float32)[:, None], d, axis=1)
    gi, gd, rec = ub.knn_bruteforce(X, k, return_stats=True)
    oi, od = oracle.knn_bruteforce(X, k, rows=(0, 200))
    assert np.array_equal(gi[:200], oi) and np.array_equal(gd[:200], od)
    assert rec < n // 100


@pytest.mark.parametrize("n,d,k,rows", [(3000, 12, 10, 128), (2500, 20, 25, 1024), (2600, 8, 100, 640), (20001, 6, 15, 4096),
                                        (17000, 5, 50, 3072), (2304, 9, 15, 2176), (2049, 9, 15, 2176)])
def test_rows_in_several_passes(ub, monkeypatch, n, d, k, rows):
    """The candidates of some rows at a time (a last pass of few rows, one row, or padding only; with and without a
    locality order): the same result as all at once."""
    X = _data(n, d, seed=n, kind="clusters")
    want = ub.knn_bruteforce(X, k)
    monkeypatch.setenv("UMAP_B200_KNN_ROWS", str(rows))
    got = ub.knn_bruteforce(X, k)
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("n,d,k,classes,sep", [(8000, 1024, 15, 50, 10), (10000, 256, 15, 50, 10), (12000, 784, 5, 10, 5),
                                               (6000, 784, 30, 50, 10)])
def test_wide_clusters_pass_their_certificates(ub, oracle, n, d, k, classes, sep):
    """Clusters so far apart that the error margin of a row holds more points than one or two lists: the splits'
    lists together hold them, and few rows are recomputed."""
    g = np.random.Generator(np.random.PCG64(n))
    X = (g.standard_normal((n, d)) + sep * g.standard_normal((classes, d))[g.integers(0, classes, n)]).astype(np.float32)
    gi, gd, rec = ub.knn_bruteforce(X, k, return_stats=True)
    oi, od = oracle.knn_bruteforce(X, k, rows=(0, 100))
    assert np.array_equal(gi[:100], oi) and np.array_equal(gd[:100], od)
    assert rec < n // 10
