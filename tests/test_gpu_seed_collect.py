"""Learned initial pools after one iteration: sorted by (distance, id), every
id once, every distance that of its pair (integer rows: exact), for pools that
take a few of a node's slots, most of them and all."""
import numpy as np
import pytest

from fastkcna_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L", [(5003, 33), (20001, 500), (3000, 1024)])
def test_learned_pools_sorted_distinct_exact(index, n, L):
    X = np.ascontiguousarray(synth.base("c2", n))
    index.upload(X)
    K = min(L, 100)
    index.nndescent(learned_seed=1, screen=1, K=K, L=L, S=8, R=60, iterations=1, search_L=min(L, 40), search_K=K, nsg_R=16)
    ids, d, cnt = index.pools()
    Xi = X.astype(np.int64)
    for i in np.r_[0, n - 1, np.arange(0, n, 97)]:
        c = int(cnt[i])
        assert 0 < c <= L
        a, b = ids[i, :c].astype(np.int64), d[i, :c]
        assert (a < n).all() and (a != i).all() and len(set(a.tolist())) == c
        assert np.array_equal(b, ((Xi[a] - Xi[i]) ** 2).sum(1).astype(np.float32))
        assert ((b[1:] > b[:-1]) | ((b[1:] == b[:-1]) & (a[1:] > a[:-1]))).all()
