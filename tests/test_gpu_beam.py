"""The beam search's batch insertion against one-by-one insertion: the oracle's
(the reference's get_neighbors) on rows without equal distances, and a
restatement below on integer rows full of them (the oracle's std::sort leaves
the order of equally far start entries open; here they go by id).  Beams of
one, odd and past a warp, rows that are no multiple of the load widths, graph
rows wider than a warp with repeated ids."""
import numpy as np
import pytest

from fastkcna_gb300 import kcna, synth

pytestmark = pytest.mark.gpu


def _one_by_one(X, g, deg, q, init, L):
    dist = lambda i: float(((X[i].astype(np.int64) - q.astype(np.int64)) ** 2).sum())
    pool = sorted((dist(i), int(i), 1) for i in init)
    seen = set(int(i) for i in init)
    k = 0
    while k < len(pool):
        nk = len(pool)
        if pool[k][2]:
            pool[k] = pool[k][:2] + (0,)
            u = pool[k][1]
            for v in g[u, : deg[u]]:
                v = int(v)
                if v in seen:
                    continue
                seen.add(v)
                d = dist(v)
                if d >= pool[-1][0]:
                    continue
                at = sum(1 for e in pool if e[0] <= d)
                pool.insert(at, (d, v, 1))
                del pool[L:]
                nk = min(nk, at)
        k = nk if nk <= k else k + 1
    return pool


@pytest.mark.parametrize("rows,d,W,L", [("c2", 128, 40, 1), ("c2", 127, 70, 33), ("c1", 32, 33, 100), ("c1", 7, 64, 31),
                                        ("c4", 258, 20, 64)])
@pytest.mark.parametrize("ties", [False, True])
def test_beam_search_inserts_as_one_by_one(index, oracle, rows, d, W, L, ties):
    n, m = 3000, 32
    X = np.ascontiguousarray(synth.base(rows, n)[:, :d])
    if ties:
        X = np.round(X * (0.02 if rows == "c2" else 2.0)).astype(np.float32)  # many equal distances
    rng = np.random.default_rng(5)
    deg = rng.integers(0, W + 1, n).astype(np.uint32)
    g = rng.integers(0, n, (n, W)).astype(np.uint32)
    g[np.arange(W)[None, :] >= deg[:, None]] = 0xFFFFFFFF
    index.upload(X)
    index.set_graph(g, deg, 0)
    Q = X[rng.integers(0, n, m)] + rng.standard_normal((m, d))
    Q = np.ascontiguousarray((np.round(Q) if ties else Q).astype(np.float32))
    init = np.stack([rng.choice(n, L, replace=False) for _ in range(m)]).astype(np.uint32)
    k = min(L, 10)
    gi, gd = index.search(Q, L, k, init)
    if not ties:
        oi, od = oracle.beam_search(X, g, deg, Q, init, L, k)
        assert np.array_equal(gi, oi) and np.array_equal(gd, od)
        return
    for i in range(m):
        pool = _one_by_one(X, g, deg, Q[i], init[i], L)[:k]
        assert gi[i].tolist() == [e[1] for e in pool] and gd[i].tolist() == [e[0] for e in pool]
