"""The join's and the merge's size classes (a warp, a small block or a large
block per node; few or many distinct survivors, the block merge above 892).
Every pool is sorted, free of repeats and of its own node, with canonical
distances; and since a join emits each pair to both ends within their radii,
which only shrink, j in i's pool nearer than j's radius means i in j's pool,
but for the S entries i started with, while no candidate buffer overflows."""
import numpy as np
import pytest

from fastkcna_gb300 import kcna, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,n,L,S,R", [("c2", 1100, 1000, 31, 200), ("c2", 4000, 501, 12, 100), ("c1", 2600, 128, 31, 40),
                                          ("c3", 1025, 1024, 20, 100), ("c1", 40, 33, 3, 8)])
@pytest.mark.parametrize("screen", [0, 1])
@pytest.mark.parametrize("iterations", [1, 3])
def test_pools_hold_every_pair_both_ways(index, monkeypatch, rows, n, L, S, R, screen, iterations):
    monkeypatch.setenv("KCNA_CAND_CAP", "8192")
    monkeypatch.setenv("KCNA_REV_CAP", "1024")
    X = synth.base(rows, n)
    index.upload(X)
    st = index.nndescent(kcna.params(K=L, L=L, S=S, R=R, iterations=iterations, delta=0.0, recall=2.0, search_L=L,
                                     search_K=L, controls=20, screen=screen))
    ids, d, cnt = index.pools()
    ti, td = index.knn_exact(np.arange(n, dtype=np.uint32), min(n - 1, 1024))
    D = np.full((n, n), np.nan, np.float32)  # canonical distances
    np.put_along_axis(D, ti.astype(np.int64), td, 1)
    cap = ids.shape[1]
    have = np.zeros((n, n), bool)
    radius = np.full(n, np.inf, np.float32)
    for i in range(n):
        c = int(cnt[i])
        p = ids[i, :c].astype(np.int64)
        assert np.unique(p).size == c and i not in p
        key = (d[i, :c].view(np.uint32).astype(np.uint64) << np.uint64(32)) | p.astype(np.uint64)
        assert (key[1:] > key[:-1]).all()
        known = ~np.isnan(D[i, p])
        assert np.array_equal(d[i, :c][known], D[i, p][known])
        have[i, p] = True
        if c == cap:
            radius[i] = d[i, c - 1]
    if sum(st["iter_cand_overflow"]):
        return  # a full buffer keeps whichever candidates came first
    for i in range(n):
        c = int(cnt[i])
        p = ids[i, :c].astype(np.int64)
        lost = (d[i, :c] < radius[p]) & ~have[p, i]
        assert lost.sum() <= S, (i, p[lost])
