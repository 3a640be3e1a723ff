"""The FP32 P2K join, whose pushes are shared among the warps in the order of the
nodes' ids: where few nodes hold the pushes, and ids go with it, every pair is still
met once (the pools are those of the same rows under other ids), and a build takes
about what it takes with the rows shuffled."""
import numpy as np
import pytest

from fastkcna_gb300 import kcna

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,hubs,W", [(4000, 40, 16), (4000, 3, 70), (3000, 700, 33), (2500, 2500, 12)])
@pytest.mark.parametrize("at", ["front", "back"])
def test_pools_do_not_depend_on_the_ids(index, monkeypatch, n, hubs, W, at):
    monkeypatch.setenv("KCNA_CAND_CAP", "8192")
    rng = np.random.default_rng(hubs)
    L = min(16, hubs)
    X = rng.standard_normal((n, 20)).astype(np.float32)
    # pools: each node's nearest of the first `hubs` rows, which so get all the pushes
    index.upload(X[:hubs] if hubs < n else X)
    if hubs < n:
        ids, dist = index.knn_queries(X, min(L + 1, hubs))
    else:
        ids, dist = index.knn_exact(np.arange(n, dtype=np.uint32), L)
    self_ = ids == np.arange(n)[:, None]
    keep = np.argsort(self_, axis=1, kind="stable")
    ids, dist = np.take_along_axis(ids, keep, 1)[:, :L].astype(np.int64), np.take_along_axis(dist, keep, 1)[:, :L]
    cnt = (~np.take_along_axis(self_, keep, 1)[:, :L]).sum(1).astype(np.uint32)
    g = np.stack([rng.choice(n, W, replace=False) for _ in range(n)])
    p = kcna.params(K=L, L=L, S=10, R=100, search_L=L, nsg_R=W, search_K=L, massq_S=10)
    out = []
    for lab in (np.arange(n) if at == "front" else np.arange(n)[::-1], rng.permutation(n)):
        inv = np.argsort(lab)  # node lab[i] is row i
        index.upload(X[inv])
        index.set_pools(lab[ids[inv]].astype(np.uint32), dist[inv], cnt[inv], p)
        index.set_graph(lab[g[inv]].astype(np.uint32), np.full(n, W, np.uint32), 0)
        comps = index.refine(1, p)
        gi, gd, gc = index.pools()
        back = np.append(inv, n).astype(np.int64)
        gi = back[np.minimum(gi[lab], n)]
        out.append((comps, gi, gd[lab], gc[lab]))
    assert out[0][0] == out[1][0] > 0
    for a, b in zip(out[0][1:], out[1][1:]):
        assert np.array_equal(a, b)


def test_rows_sorted_by_norm(index):
    rng = np.random.default_rng(5)
    n = 20000
    X = rng.standard_normal((n, 400)).astype(np.float32) * np.linspace(0.1, 3, n, dtype=np.float32)[:, None]
    p = kcna.params(K=100, L=100, S=10, R=100, iterations=5, search_L=40, nsg_R=32, search_K=100, recall=2.0, delta=0.0)
    ms = []
    for rows in (X, X[rng.permutation(n)]):
        index.upload(rows)
        ms.append(min(index.build("nsg", p)["phase_ms"]["p2k"] for _ in range(4)))
    assert ms[0] < 2.0 * ms[1], ms
