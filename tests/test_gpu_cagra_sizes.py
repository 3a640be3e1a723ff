"""The rank prune on both sides of a warp per node (K = 64) and of the powers of
two that size its tables, against the oracle; short pools among them."""
import numpy as np
import oracle_py
import pytest

from fastkcna_gb300 import kcna

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [2, 62, 64, 66, 100, 128, 130, 256, 514])
def test_rank_prune_equals_oracle(index, oracle, K):
    n, d = 900, 12
    rng = np.random.default_rng(K)
    X = rng.integers(-200, 201, (n, d)).astype(np.float32)
    index.upload(X)
    ids, dist = index.knn_exact(np.arange(n, dtype=np.uint32), K)
    cnt = np.full(n, K, np.uint32)
    cnt[::9] = np.maximum(K // 2 + 1, 2)
    kw = dict(K=K, L=K, S=10, R=100, iterations=1, search_L=min(K, 40), nsg_R=min(K, 32), search_K=K)
    p = kcna.params(**kw)
    index.set_pools(ids, dist, cnt, p)
    index.prune("cagra", p)
    g, deg, _ = index.graph()
    oi, _, odeg = oracle.prune(oracle_py.KCNA_CAGRA, X, oracle_py.params(**kw), ids, dist, cnt, K // 2 + 1)
    assert np.array_equal(deg, odeg)
    live = np.arange(K // 2 + 1) < deg[:, None]
    assert np.array_equal(g[:, : K // 2 + 1][live], oi[live])
