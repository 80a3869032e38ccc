"""smooth_knn at the edges of its lanes per row (16 up to 128 rows per SM, 4 up to 256, then 1), against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL_TOL = 1e-5


@pytest.mark.parametrize("per_sm,extra", [(128, 0), (128, 1), (256, 0), (256, 1)])
@pytest.mark.parametrize("k", [2, 5, 16, 33])
def test_sigmas_rhos_match_oracle(ub, oracle, k, per_sm, extra):
    import torch
    n = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + extra
    g = np.random.Generator(np.random.PCG64(k))
    dist = np.sort(g.gamma(2.0, 1.0, (n, k)).astype(np.float32), axis=1)
    dist[::3, 0] = 0.0
    dist[::50] = 1.5            # every distance the same
    dist[::77] = 0.0            # no distance above 0
    idx = ((np.arange(n)[:, None] + np.arange(k)[None, :] * 11) % n).astype(np.uint32)
    cfg = ub.UmapConfig()
    cfg.graph.n_neighbors = k
    s, r = ub.Umap(cfg).learn_manifold(n, idx, dist).sigmas_rhos()
    so, ro = oracle.learn_manifold(idx, dist, oracle.OracleConfig(n_neighbors=k)).sigmas_rhos()
    assert np.array_equal(r, ro)
    assert np.allclose(s, so, rtol=REL_TOL, atol=0)
