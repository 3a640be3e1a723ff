"""The FP32 join's size classes: rows a few of which are everyone's neighbours
(hubs), so that their nodes join far more rows than the others.  Without a full
candidate buffer every pair within both radii is held both ways, whichever kernel
joined it; and the pairs per row show that some node had more than 64 rows (one
of r rows has at most (r - 1) / 2 per row)."""
import numpy as np
import pytest

from fastkcna_gb300 import kcna

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,hubs,L,S,R,iterations", [(600, 100, 60, 31, 100, 2), (600, 30, 100, 12, 200, 3), (1000, 6, 60, 3, 400, 5),
                                                     (1000, 20, 100, 6, 400, 4)])
def test_nodes_of_many_rows(index, monkeypatch, n, hubs, L, S, R, iterations):
    monkeypatch.setenv("KCNA_CAND_CAP", "8192")
    monkeypatch.setenv("KCNA_REV_CAP", "1024")
    X = np.random.default_rng(4).standard_normal((n, 32)).astype(np.float32)
    X /= np.linalg.norm(X, axis=1)[:, None]
    X[:hubs] *= 0.2
    index.upload(X)
    done = []
    for it in (iterations - 1, iterations):
        st = index.nndescent(kcna.params(K=L, L=L, S=S, R=R, iterations=it, delta=0.0, recall=2.0, search_L=L, search_K=L,
                                         controls=20))
        done.append((st["n_comps"], st["join_rows"]))
    assert sum(st["iter_cand_overflow"]) == 0
    assert (done[1][0] - done[0][0]) / (done[1][1] - done[0][1]) > 31.5, done
    ids, dist, cnt = index.pools()
    ti, td = index.knn_exact(np.arange(n, dtype=np.uint32), n - 1)
    D = np.zeros((n, n), np.float32)
    np.put_along_axis(D, ti.astype(np.int64), td, 1)
    have = np.zeros((n, n), bool)
    radius = np.full(n, np.inf, np.float32)
    for i in range(n):
        c = int(cnt[i])
        p = ids[i, :c].astype(np.int64)
        assert np.unique(p).size == c and i not in p
        assert np.array_equal(dist[i, :c], D[i, p]) and (dist[i, 1:c] >= dist[i, : c - 1]).all()
        have[i, p] = True
        if c == ids.shape[1]:
            radius[i] = dist[i, c - 1]
    for i in range(n):
        p = ids[i, : cnt[i]].astype(np.int64)
        lost = (dist[i, : cnt[i]] < radius[p]) & ~have[p, i]
        assert lost.sum() <= S, (i, p[lost])
