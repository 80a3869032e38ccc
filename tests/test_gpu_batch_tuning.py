"""The batch tuner's cache: a search that ended early, because no row was longer than its task, says nothing of
batches with longer rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(ub, hub):
    """Two instances of 1,501 points and 10 neighbours; with `hub`, all of them also neighbours of point 0."""
    n, k = 1501, 10
    g = np.random.Generator(np.random.PCG64(4))
    idx = (np.arange(n)[:, None] + 1 + np.arange(k)[None, :] * 3) % n
    if hub:
        idx[1:, 0] = np.where((idx[1:] == 0).any(1), idx[1:, 0], 0)
    dist = np.sort(g.uniform(0.5, 2.0, (n, k)).astype(np.float32), axis=1)
    init = g.uniform(-1, 1, (n, 2)).astype(np.float32)
    cfg = ub.UmapConfig()
    cfg.graph.n_neighbors = k
    two = [np.concatenate([a, a]) for a in (idx.astype(np.uint32), dist, init)]
    return ub.Optimizer.batch(cfg, [0, n, 2 * n], *two, 100)


def test_early_end_is_not_kept_for_longer_rows(ub, monkeypatch, capfd):
    monkeypatch.setenv("UMAP_B200_LOG", "1")
    searches = []
    for hub in (False, False, True, True, False):
        capfd.readouterr()
        opt = _batch(ub, hub)
        searches.append(capfd.readouterr().err.count("autotune"))
        assert np.isfinite(opt.embedding()).all()
    assert searches == [1, 0, 1, 0, 0]


def test_any_dimension_kernel_tries_smaller_blocks(ub):
    """300 instances of 300 points in 5-D at a small rate: blocks of 128 threads spread the tasks over more SMs and
    take a quarter off the epoch, so the tuner finds them."""
    g = np.random.Generator(np.random.PCG64(2))
    n, k, m = 300, 10, 300
    idx = (np.arange(n)[:, None] + np.arange(k)[None, :] * 7) % n
    dist = np.sort(g.uniform(0.1, 2.0, (m * n, k)).astype(np.float32), axis=1)
    dist[:, 0] = 0.0
    cfg = ub.UmapConfig(n_components=5)
    cfg.graph.n_neighbors = k
    cfg.optimization.learning_rate = 0.005
    init = g.uniform(-1, 1, (m * n, 5)).astype(np.float32)
    opt = ub.Optimizer.batch(cfg, np.arange(m + 1) * n, np.tile(idx.astype(np.uint32), (m, 1)), dist, init, 60)
    assert "anydim" in opt.layout()["kernel"] and opt.tuning()[1] == 128
