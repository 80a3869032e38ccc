"""Which epoch kernel a layout takes (by size, columns and learning rate), and that fits at small rates,
which hardly change from run to run, stay where the lane-per-task kernels put them."""
import os
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden"))
import make_small_rate as small  # noqa: E402
from test_gpu_epoch_kernels import _config, _spread, _stars, _steps  # noqa: E402


def _layout(ub, n, dim, rate, generic=False, k=15):
    g = np.random.Generator(np.random.PCG64(n))
    idx = (np.arange(n)[:, None] + np.arange(k)[None, :] * 7) % n
    dist = np.sort(g.uniform(0.1, 2.0, (n, k)).astype(np.float32), axis=1)
    dist[:, 0] = 0.0
    cfg = ub.UmapConfig(n_components=dim)
    cfg.optimization.learning_rate = rate
    init = g.uniform(-1, 1, (n, dim)).astype(np.float32)
    mt = ub.MetricType.Generic if generic else ub.MetricType.Euclidean
    opt = ub.Optimizer(ub.Umap(cfg).learn_manifold(n, idx.astype(np.uint32), dist), init, 20, cfg, mt)
    return opt.layout()


@pytest.mark.parametrize("n,dim,rate,generic,kernel", [
    (500, 2, 0.006, False, "sgd_epoch_kernel2<2, false, 8, 4, true>"),
    (500, 2, 0.01, False, "sgd_epoch_kernel2<2, false, 8, 4, true>"),
    (500, 1, 0.03, False, "sgd_epoch_pool<1, false>"),
    (20000, 2, 0.009, False, "sgd_epoch_kernel2<2, false, 8, 4, true>"),
    (20000, 2, 0.01, False, "sgd_epoch_pool<2, false>"),
    (20000, 2, 0.01, True, "sgd_epoch_kernel2<2, true, 4, 5, true>"),
    (20000, 2, 1.0, True, "sgd_epoch_pool<2, true>"),
    (2000, 3, 0.02, False, "sgd_epoch_kernel2<3, false, 4, 5, true>"),
    (2000, 4, 0.03, False, "sgd_epoch_pool<4, false>"),
    (2000, 5, 0.02, False, "sgd_epoch_anydim<false>"),
    (2000, 7, 0.03, False, "sgd_epoch_rows<7>"),
    (2000, 8, 1.0, False, "sgd_epoch_anydim<false>"),
])
def test_kernel_by_rate(ub, n, dim, rate, generic, kernel):
    assert _layout(ub, n, dim, rate, generic)["kernel"] == kernel


@pytest.mark.parametrize("name", list(small.CASES))
def test_small_rate_fits_agree(ub, name):
    """Four runs an input against the recorded mean, each distance in units of a recorded run's.  Runs
    of the same kernels have their median near 1 (0.9 to 1.6 over machines), the pooled kernel's at 2.3 to 3.6."""
    z = np.load(os.path.join(os.path.dirname(small.__file__), "small_rate.npz"))
    ratio = [small.distance(small.fit(ub, name, seed), z[f"{name}_{seed}_mean"]) / float(z[f"{name}_{seed}_own"])
             for seed in range(small.CASES[name][-1]) for _ in range(4)]
    assert np.median(ratio) <= 2.0, np.round(sorted(ratio), 2)


@pytest.mark.parametrize("chunk", ["64", "16"])
@pytest.mark.parametrize("neg", [5, 20])
@pytest.mark.parametrize("a,b,dim", [("lane", "pool", 2), ("lane", "pool", 3), ("lane", "pool", 4), ("rows", "pool", 5),
                                     ("rows", "pool", 6), ("rows", "pool", 7), ("dram", "lane", 2), ("dram", "lane", 1)])
def test_forced_kernels_draw_the_same_negatives(ub, monkeypatch, a, b, dim, neg, chunk):
    """Two kernels on the same layout (rows: against the pooled kernel in 2-D, its other columns zero; dram: against
    the lane kernel on interleaved entries) draw the same negatives.  At rate 1e-4 they agree within 1e-4, for the
    reason given at test_negatives_are_the_same_draws."""
    idx, dist, init = _stars(3)
    monkeypatch.setenv("UMAP_B200_CHUNK", chunk)
    monkeypatch.setenv("UMAP_B200_SGD_LANE_MAJOR", "0" if a == "dram" else "1")
    out = []
    for kernel, d in ((a, dim), (b, 2 if a == "rows" else dim)):
        monkeypatch.setenv("UMAP_B200_SGD_KERNEL", kernel)
        e, layout = _steps(ub, _config(ub, d, 12, neg, 1e-4), idx, dist, _spread(init, d), 12, (1,) * 6)
        assert {"lane": "kernel2", "any": "anydim"}.get(kernel, kernel) in layout["kernel"]
        out.append(e if d == 1 else e[:, [0, -1]])
        assert np.abs(e[:, 1:-1]).max(initial=0.0) == 0.0
    assert np.abs(out[0] - out[1]).max() <= 1e-4


@pytest.mark.parametrize("neg", [5, 20])
@pytest.mark.parametrize("a,b,dim", [("pool", "lane", 2), ("pool", "lane", 3), ("rows", "any", 5)])
def test_batch_kernels_draw_the_same_negatives(ub, monkeypatch, a, b, dim, neg):
    """The same for two instances of a batch, whose rows of 33 to 40 entries cross a window of 32."""
    monkeypatch.setenv("UMAP_B200_AUTOTUNE", "0")
    monkeypatch.setenv("UMAP_B200_CHUNK", "64")
    parts = [_stars(5), _stars(6)]
    n = len(parts[0][0])
    idx, dist, init = (np.concatenate(x) for x in zip(*parts))
    out = []
    for kernel in (a, b):
        monkeypatch.setenv("UMAP_B200_SGD_KERNEL", kernel)
        opt = ub.Optimizer.batch(_config(ub, dim, 12, neg, 1e-4), [0, n, 2 * n], idx, dist, _spread(init, dim), 12)
        assert {"lane": "kernel2", "any": "anydim"}.get(kernel, kernel) in opt.layout()["kernel"]
        for _ in range(6):
            opt.step_epochs(1)
        out.append(opt.embedding())
    assert np.abs(out[0] - out[1]).max() <= 1e-4


@pytest.mark.parametrize("kernel", ["lane", "pool", "dram"])
def test_forced_kernels_quality_with_split_rows(ub, oracle, monkeypatch, kernel):
    """The 20,000-point sheet-initialised roll of test_embedding_quality_on_a_structured_manifold, in a renamed layout
    whose rows of more than 16 edges are cut: recall and fuzzy cross-entropy in the oracle's band."""
    from test_gpu_parity import _assert_quality, _oracle_scores
    from umap_b200 import quality as Q
    from umap_b200 import workloads as W
    X, t = W.swiss_roll(20000, seed=3)
    idx, dist = W.knn_exact_numpy(X, 15)
    init = np.stack([t, X[:, 1]], 1).astype(np.float32)
    cfg = ub.UmapConfig()
    cfg.optimization.n_epochs = 200
    rec_o, ce_o, (head, tail, w), (a, b) = _oracle_scores(oracle, idx, dist, init, 200)
    monkeypatch.setenv("UMAP_B200_SGD_KERNEL", kernel)
    monkeypatch.setenv("UMAP_B200_RELABEL", "1")
    res = []
    for seed in (1, 2, 3):
        opt = ub.Optimizer(ub.Umap(cfg).learn_manifold(20000, idx, dist), init, 200, cfg)
        assert {"lane": "kernel2"}.get(kernel, kernel) in opt.layout()["kernel"] and opt.layout()["renamed"]
        assert opt.tuning()[0] == 16 and np.bincount(head).max() > 16
        opt.set_seed(seed)
        opt.step_epochs(200)
        e = opt.embedding()
        res.append((Q.knn_recall(e, idx), Q.fuzzy_cross_entropy(e, head, tail, w, a, b)))
    _assert_quality(res, rec_o, ce_o, f"roll 20k, {kernel}")
