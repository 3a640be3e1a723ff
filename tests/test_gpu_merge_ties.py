"""NN-descent's merge on few-valued rows, whose pools hold long runs of equal
distances: strictly sorted by (distance, id) with exact distances, every pair
held both ways, and merges that cost about what those of nearly the same rows
without equal distances do."""
import numpy as np
import pytest

from fastkcna_gb300 import kcna

pytestmark = pytest.mark.gpu


def _params(L, S, R, iterations, screen=0):
    return kcna.params(K=L, L=L, S=S, R=R, iterations=iterations, delta=0.0, recall=2.0, search_L=L, search_K=L, controls=20,
                       screen=screen)


@pytest.mark.parametrize("levels,n,d,L,S,R", [(2, 3000, 48, 200, 10, 40), (2, 2500, 12, 500, 12, 40), (3, 3000, 20, 300, 12, 40)])
@pytest.mark.parametrize("screen", [0, 1])
@pytest.mark.parametrize("iterations", [1, 4])
def test_pools_of_few_valued_rows(index, monkeypatch, levels, n, d, L, S, R, screen, iterations):
    monkeypatch.setenv("KCNA_CAND_CAP", "8192")
    monkeypatch.setenv("KCNA_REV_CAP", "1024")
    X = np.random.default_rng(4).integers(0, levels, (n, d)).astype(np.float32)
    index.upload(X)
    st = index.nndescent(_params(L, S, R, iterations, screen))
    assert sum(st["iter_cand_overflow"]) == 0  # nothing below holds where a buffer fills
    ids, dist, cnt = index.pools()
    have = np.zeros((n, n), bool)
    radius = np.full(n, np.inf, np.float32)
    for i in range(n):
        c = int(cnt[i])
        p = ids[i, :c].astype(np.int64)
        assert i not in p and np.array_equal(dist[i, :c], ((X[p] - X[i]) ** 2).sum(1))
        key = dist[i, :c].astype(np.int64) * n + p
        assert (key[1:] > key[:-1]).all()
        have[i, p] = True
        if c == ids.shape[1]:
            radius[i] = dist[i, c - 1]
    for i in range(n):
        p = ids[i, : cnt[i]].astype(np.int64)
        lost = (dist[i, : cnt[i]] < radius[p]) & ~have[p, i]
        assert lost.sum() <= S, (i, p[lost])  # the S entries it started with


def test_equal_distances_do_not_slow_the_merge(index):
    n, d, K = 40000, 64, 500
    rng = np.random.default_rng(8)
    X = rng.integers(0, 2, (n, d)).astype(np.float32)
    p = _params(K, 10, 100, 6)
    ms = []
    for rows in (X, X + 1e-3 * rng.standard_normal((n, d)).astype(np.float32)):
        index.upload(rows)
        ms.append(min(sum(index.nndescent(p)["iter_merge_ms"][2:]) for _ in range(4)))
    assert ms[0] < 1.7 * ms[1], ms
