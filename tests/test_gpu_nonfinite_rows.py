"""Rows with infinite, NaN or very distant coordinates: the epoch kernels keep the rule's gates (a repulsion moves
only where its coefficient is above 0, an attraction's coefficient is 0 at a NaN distance), so such a row spoils
the same coordinates as in the oracle and no others."""
import numpy as np
import pytest

from test_gpu_epoch_kernels import _config, _spread, _stars

pytestmark = pytest.mark.gpu

KERNELS = [("pool", 1), ("pool", 2), ("pool", 3), ("pool", 4), ("lane", 1), ("lane", 2), ("lane", 3), ("dram", 1), ("dram", 2),
           ("rows", 5), ("rows", 7), ("any", 5), ("any", 8)]


def _run(ub, oracle, monkeypatch, kernel, dim, idx, dist, init, neg, rate):
    monkeypatch.setenv("UMAP_B200_SGD_KERNEL", kernel)
    monkeypatch.setenv("UMAP_B200_CHUNK", "64")
    cfg = _config(ub, dim, 8, neg, rate)
    opt = ub.Optimizer(ub.Umap(cfg).learn_manifold(len(idx), idx, dist), init, 8, cfg)
    ocfg = oracle.OracleConfig(n_neighbors=idx.shape[1], negative_sample_rate=neg, n_epochs=8, learning_rate=rate,
                               symmetrize=False, n_components=dim)
    oo = oracle.Optimizer(oracle.learn_manifold(idx, dist, ocfg), init, 8, ocfg, seed=1)
    assert np.array_equal(opt.embedding(), oo.embedding(), equal_nan=True)
    opt.step_epochs(8)
    oo.step_epochs(8)
    return opt.embedding(), oo.embedding()


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("kernel,dim", KERNELS)
def test_bad_rows_drawn_as_negatives(ub, oracle, monkeypatch, kernel, dim, bad):
    """Every vertex without an edge has a bad first coordinate: half of all draws.  Each draw leaves the head
    where it is, so all other rows stay finite."""
    idx, dist, init = _stars(7)
    init = _spread(init, dim)
    n = len(idx)
    linked = np.unique(np.concatenate([np.arange(75), idx[idx < n]]))
    lone = np.setdiff1d(np.arange(n), linked)
    assert len(lone) > n // 3
    init[lone, 0] = bad
    got, want = _run(ub, oracle, monkeypatch, kernel, dim, idx, dist, init, 5, 0.1)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    assert np.isfinite(got[linked]).all()


@pytest.mark.parametrize("bad", [np.inf, np.nan, 1e16])
@pytest.mark.parametrize("kernel,dim", KERNELS)
def test_bad_tails(ub, oracle, monkeypatch, kernel, dim, bad):
    """A leaf of every fifth centre has a bad first coordinate (1e16: beside an infinite lone row, which keeps the
    column from being rescaled; at that distance the coefficient is 0).  No negatives, whole rows: the sequence of
    moves is the oracle's."""
    idx, dist, init = _stars(8)
    init = _spread(init, dim)
    init[75 + np.arange(0, 75, 5) * 40, 0] = bad
    if np.isfinite(bad):
        init[-1, 0] = np.inf
        idx[74, -1] = 0xFFFFFFFF
    got, want = _run(ub, oracle, monkeypatch, kernel, dim, idx, dist, init, 0, 0.1)
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    ok = np.isfinite(want)
    assert np.allclose(got[ok], want[ok], rtol=1e-4, atol=1e-4)
