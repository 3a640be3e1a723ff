"""The rank prune and the FP32 prune on both sides of the node counts from which a
warp per node, and batches in shared memory, pay; against the oracle.  And the rank
prune of few nodes at a small K costs no more than at a larger one."""
import time

import numpy as np
import oracle_py
import pytest

from fastkcna_gb300 import kcna

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,K", [(1023, 8), (1024, 8), (767, 8), (1535, 16), (1536, 16), (6143, 64), (6144, 64), (6300, 62), (6400, 66)])
def test_rank_prune_equals_oracle(index, oracle, n, K):
    d = 12
    rng = np.random.default_rng(n + K)
    X = rng.integers(-200, 201, (n, d)).astype(np.float32)
    X[:5] //= 8  # in many pools: long reverse segments
    index.upload(X)
    ids, dist = index.knn_exact(np.arange(n, dtype=np.uint32), K)
    cnt = np.full(n, K, np.uint32)
    cnt[::9] = max(K // 2 + 1, 2)
    kw = dict(K=K, L=K, S=10, R=100, iterations=1, search_L=min(K, 40), nsg_R=min(K, 32), search_K=K)
    p = kcna.params(**kw)
    index.set_pools(ids, dist, cnt, p)
    index.prune("cagra", p)
    g, deg, _ = index.graph()
    oi, _, odeg = oracle.prune(oracle_py.KCNA_CAGRA, X, oracle_py.params(**kw), ids, dist, cnt, K // 2 + 1)
    assert np.array_equal(deg, odeg)
    live = np.arange(K // 2 + 1) < deg[:, None]
    assert np.array_equal(g[:, : K // 2 + 1][live], oi[live])


@pytest.mark.parametrize("kind", [1, 3, 4])
@pytest.mark.parametrize("n,d,k,R", [(4096, 32, 33, 4), (4095, 61, 60, 32), (4100, 61, 200, 5), (1536, 96, 260, 128), (1535, 96, 100, 40),
                                     (1600, 189, 70, 36), (1600, 192, 100, 40), (1600, 96, 2, 1), (1600, 64, 90, 37)])
def test_warp_prune_equals_oracle(index, oracle, kind, n, d, k, R):
    rng = np.random.default_rng(d + k)
    X = rng.standard_normal((n, d)).astype(np.float32)
    X /= np.linalg.norm(X, axis=1, keepdims=True)
    X[50:90] = X[7]
    X[90:130] *= np.float32(0.25)
    index.upload(X)
    ids, dist = index.knn_exact(np.arange(n, dtype=np.uint32), k)
    cnt = np.full(n, k, np.uint32)
    cnt[::7] = 1
    cnt[3::7] = max(1, k // 3)
    kw = dict(K=k, L=k, S=10, R=100, iterations=1, search_L=40, nsg_R=R, search_K=k, tau=0.02, angle=60.0)
    kp = kcna.params(**kw)
    index.set_pools(ids, dist, cnt, kp)
    index.prune({1: "nsg", 3: "taumng", 4: "alphapg"}[kind], kp)
    g, deg, _ = index.graph()
    oi, _, odeg = oracle.prune(kind, X, oracle_py.params(**kw), ids, dist, cnt, g.shape[1])
    assert np.array_equal(deg, odeg)
    assert np.array_equal(g, oi)


def _time(f, reps=60):
    f()
    t = []
    for _ in range(reps):
        t0 = time.perf_counter()
        f()
        t.append(time.perf_counter() - t0)
    return sorted(t)[reps // 6]


def test_rank_prune_of_few_nodes(index):
    """K = 64 (a warp per node on large bases) against the four times as many
    look-ups of K = 128 (a block per node)."""
    n = 600
    X = np.random.default_rng(1).standard_normal((n, 32)).astype(np.float32)
    index.upload(X)
    ids, dist = index.knn_exact(np.arange(n, dtype=np.uint32), 128)
    t = []
    for K in (64, 128):
        p = kcna.params(K=K, L=128, search_K=K, search_L=128)
        index.set_pools(ids, dist, np.full(n, 128, np.uint32), p)
        t.append(_time(lambda: index.prune("cagra", p)))
    assert t[0] < 1.02 * t[1], t
