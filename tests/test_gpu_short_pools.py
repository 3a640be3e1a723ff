"""NN-descent whose pools are shorter than the S entries a node starts with: pools
of at most L entries, sorted, without repeats, with canonical distances, and ids of
rows throughout.  No pools at all are refused."""
import numpy as np
import pytest

from fastkcna_gb300 import kcna

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L,S,K,sl", [(52, 12, 30, 12, 12), (700, 5, 31, 9, 40), (1000, 1, 10, 3, 3), (24, 10, 12, 60, 4),
                                        (300, 30, 31, 30, 30), (300, 31, 31, 31, 31)])
@pytest.mark.parametrize("screen", [0, 1])
@pytest.mark.parametrize("iterations", [1, 4])
def test_pools_shorter_than_their_start(index, n, L, S, K, sl, screen, iterations):
    X = np.random.default_rng(n).standard_normal((n, 24)).astype(np.float32)
    index.upload(X)
    index.nndescent(kcna.params(K=K, L=L, S=S, R=20, iterations=iterations, search_L=sl, search_K=sl, recall=2.0, delta=0.0,
                                controls=10, screen=screen))
    ids, d, cnt = index.pools()
    ti, td = index.knn_exact(np.arange(n, dtype=np.uint32), n - 1)
    D = np.zeros((n, n), np.float32)
    np.put_along_axis(D, ti.astype(np.int64), td, 1)
    assert (cnt <= min(L, n - 1)).all() and (cnt > 0).all()
    for i in range(n):
        p = ids[i, : cnt[i]].astype(np.int64)
        assert (p < n).all() and i not in p and np.unique(p).size == p.size
        assert np.array_equal(d[i, : cnt[i]], D[i, p]) and (np.diff(d[i, : cnt[i]]) >= 0).all()


def test_no_pools(index):
    index.upload(np.random.default_rng(1).standard_normal((50, 8)).astype(np.float32))
    with pytest.raises(kcna.KcnaArgError):
        index.nndescent(kcna.params(K=5, L=0, S=3, search_L=5, search_K=5))
