"""The SGD epoch kernels on star graphs: every centre has its own leaves and a leaf has no edges, so
a centre's firings form one sequence that no other row touches.  Degrees 1 to 40 cross the kernels'
windows of 16 and 32 entries; 75 centres leave slices, blocks and pools partly empty."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CENTRES, K = 75, 40


def _stars(seed=0):
    """kNN arrays of CENTRES stars (directed graph, centre i keeps 1 + i * 39 // 74 leaves) and a 2-D init."""
    g = np.random.Generator(np.random.PCG64(seed))
    n = CENTRES * (1 + K)
    idx = np.full((n, K), 0xFFFFFFFF, np.uint32)
    dist = np.sort(g.uniform(0.5, 2.0, (n, K)).astype(np.float32), axis=1)
    for i in range(CENTRES):
        deg = 1 + i * (K - 1) // (CENTRES - 1)
        idx[i, :deg] = CENTRES + i * K + np.arange(deg)
    init = g.uniform(-10, 10, (n, 2)).astype(np.float32)
    return idx, dist, init


def _config(ub, dim, epochs, neg, rate):
    cfg = ub.UmapConfig(n_components=dim)
    cfg.graph.n_neighbors = K
    cfg.graph.symmetrize = False
    cfg.optimization.negative_sample_rate = neg
    cfg.optimization.n_epochs = epochs
    cfg.optimization.learning_rate = rate
    return cfg


def _steps(ub, cfg, idx, dist, init, epochs, steps):
    opt = ub.Optimizer(ub.Umap(cfg).learn_manifold(len(idx), idx, dist), init, epochs, cfg)
    for s in steps:
        opt.step_epochs(s)
    return opt.embedding(), opt.layout()


KERNELS = [("pool", 1), ("pool", 2), ("pool", 3), ("pool", 4), ("dram", 1), ("dram", 2), ("", 5), ("", 6), ("", 7), ("", 8), ("", 33)]


def _spread(init, dim):
    """The 2-D init in the first and last of `dim` columns, the others zero (dim 1: its first column)."""
    if dim == 1:
        return np.ascontiguousarray(init[:, :1])
    wide = np.zeros((len(init), dim), np.float32)
    wide[:, 0], wide[:, -1] = init[:, 0], init[:, 1]
    return wide


@pytest.mark.parametrize("kernel,dim", KERNELS)
def test_sequential_rows_match_oracle(ub, oracle, monkeypatch, kernel, dim):
    """No negatives, whole rows: the same sequence of attractions as the oracle's, 12 epochs at rate
    0.1.  Up to 480 steps of a contraction with about 1e-6 relative error each: within 1e-4."""
    idx, dist, init = _stars()
    init = _spread(init, dim)
    monkeypatch.setenv("UMAP_B200_CHUNK", "64")
    if kernel:
        monkeypatch.setenv("UMAP_B200_SGD_KERNEL", kernel)
    got, layout = _steps(ub, _config(ub, dim, 12, 0, 0.1), idx, dist, init, 12, (7, 5))
    assert kernel in layout["kernel"]
    ocfg = oracle.OracleConfig(n_neighbors=K, negative_sample_rate=0, n_epochs=12, learning_rate=0.1, symmetrize=False,
                               n_components=dim)
    oo = oracle.Optimizer(oracle.learn_manifold(idx, dist, ocfg), init, 12, ocfg, seed=1)
    x0 = oo.embedding()
    oo.step_epochs(7)
    oo.step_epochs(5)
    want = oo.embedding()
    assert np.allclose(got, want, rtol=1e-4, atol=1e-4), np.abs(got - want).max()
    assert np.abs(want - x0).max() > 1e-2


@pytest.mark.parametrize("chunk", ["64", "16"])
@pytest.mark.parametrize("neg", [5, 20])
@pytest.mark.parametrize("kernel,dim", [k for k in KERNELS if k[0] != "dram" and k[1] > 1 and k != ("pool", 2)])
def test_negatives_are_the_same_draws(ub, monkeypatch, kernel, dim, neg, chunk):
    """The kernels draw the same negatives (same entry, epoch and pair), so a fit with two live
    columns, the others all zero, moves them as the pooled 2-D kernel does.  At rate 1e-4 a
    racing read differs by one move (4e-4 at most), which changes a later move by under 1e-4 of
    it times the repulsion's slope (below 1,800): within 1e-4."""
    idx, dist, init = _stars(3)
    monkeypatch.setenv("UMAP_B200_CHUNK", chunk)
    monkeypatch.setenv("UMAP_B200_SGD_KERNEL", "pool")
    want, _ = _steps(ub, _config(ub, 2, 12, neg, 1e-4), idx, dist, init, 12, (1,) * 6)
    monkeypatch.setenv("UMAP_B200_SGD_KERNEL", kernel)
    got, layout = _steps(ub, _config(ub, dim, 12, neg, 1e-4), idx, dist, _spread(init, dim), 12, (1,) * 6)
    assert kernel in layout["kernel"]
    assert np.abs(got[:, 1:-1]).max(initial=0.0) == 0.0
    assert np.abs(got[:, [0, -1]] - want).max() <= 1e-4
