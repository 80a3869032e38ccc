"""Writes tests/golden/small_rate.npz: fits at small learning rates, where a layout hardly changes from
run to run, as the library's lane-per-task epoch kernels produced them.  Per case of CASES: the
mean embedding of RUNS fits and, per input, the median distance of a run from it (relative
2-norms).  tests/test_gpu_epoch_choice.py holds later builds to these.

Usage, on the GPU: python tests/golden/make_small_rate.py OUT.npz [PACKAGE_PARENT]
"""
from __future__ import annotations

import os
import sys

import numpy as np

# 5-D fits are not held: sgd_epoch_anydim's runs agree to 1e-5 within a machine and differ by 4e-5 between
# machines.
# name: (points, components, epochs, learning rate, inputs)
CASES = {"2d": (500, 2, 500, 0.006, 6), "3d": (1000, 3, 200, 0.006, 3)}
RUNS = 16


def inputs(n, comp, seed, k=15):
    """Six Gaussian clusters in 8-D, exact kNN with the point itself first, the first columns as init."""
    g = np.random.Generator(np.random.PCG64(seed))
    x = g.standard_normal((n, 8)) + 5.0 * g.standard_normal((6, 8))[g.integers(0, 6, n)]
    d = np.zeros((n, n))
    for c in range(8):
        d += (x[:, None, c] - x[None, :, c]) ** 2
    np.fill_diagonal(d, -1.0)
    idx = np.argsort(d, axis=1, kind="stable")[:, :k]
    dist = np.sqrt(np.maximum(np.take_along_axis(d, idx, 1), 0.0))
    return idx.astype(np.uint32), dist.astype(np.float32), np.ascontiguousarray(x[:, :comp], np.float32)


def fit(ub, name, seed):
    n, comp, epochs, rate, _ = CASES[name]
    cfg = ub.UmapConfig(n_components=comp)
    cfg.optimization.n_epochs, cfg.optimization.learning_rate = epochs, rate
    return ub.Umap(cfg).fit(n, *inputs(n, comp, seed)).embedding()


def distance(a, mean):
    return float(np.linalg.norm(a - mean) / np.linalg.norm(mean))


if __name__ == "__main__":
    root = os.path.dirname(os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    sys.path.insert(0, sys.argv[2] if len(sys.argv) > 2 else os.path.join(root, "umap-rs_b200"))
    import umap_b200 as ub
    out = {}
    for name, case in CASES.items():
        for seed in range(case[-1]):
            runs = np.stack([fit(ub, name, seed) for _ in range(RUNS)]).astype(np.float64)
            mean = runs.mean(0)
            out[f"{name}_{seed}_mean"] = mean.astype(np.float32)
            out[f"{name}_{seed}_own"] = np.float32(np.median([distance(r, mean) for r in runs]))
    np.savez_compressed(sys.argv[1], **out)
