"""Union and edge-list kernels at the edges of their lane groups: rows that keep 0, 1, 15, 16, 17, 31, 32, 33
neighbours, and a hub whose transposed row is longer than any group."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

REL_TOL = 1e-5


def _knn(n, k, seed):
    """Vertex i keeps i % (k + 1) neighbours, vertex 0 always among them; the rest are sentinels."""
    g = np.random.Generator(np.random.PCG64(seed))
    idx = np.full((n, k), 0xFFFFFFFF, np.uint32)
    dist = np.sort(g.uniform(0.1, 3.0, (n, k)).astype(np.float32), axis=1)
    for i in range(n):
        deg = i % (k + 1)
        if deg:
            idx[i, :deg] = np.concatenate([[0], 1 + g.choice(n - 1, deg - 1, replace=False)])
    return idx, dist


@pytest.mark.parametrize("mix", [0.0, 0.25, 1.0])
@pytest.mark.parametrize("n,k", [(40, 2), (301, 15), (301, 16), (300, 17), (299, 32), (67, 33), (400, 64)])
def test_union_matches_oracle(ub, oracle, n, k, mix):
    idx, dist = _knn(n, k, n + k)
    cfg = ub.UmapConfig()
    cfg.graph.n_neighbors = k
    cfg.graph.set_op_mix_ratio = mix
    got = ub.Umap(cfg).learn_manifold(n, idx, dist).graph()
    ptr, ind, data = oracle.learn_manifold(idx, dist, oracle.OracleConfig(n_neighbors=k, set_op_mix_ratio=mix)).graph()
    assert np.array_equal(got.indptr, ptr)
    assert np.array_equal(got.indices, ind)
    # two memberships within REL_TOL of the oracle's, in a form whose derivatives in them are at most 1
    assert np.allclose(got.data, data, rtol=0, atol=2 * REL_TOL)
