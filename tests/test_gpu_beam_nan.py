"""Beam search with rows at a NaN distance: such a row is farther than any other,
so as a start entry it gives way to every neighbour met, and as a neighbour it
enters only where nothing else would.  Against one-by-one insertion on integer
rows, whose distances are exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _one_by_one(X, g, q, init, L):
    far = np.uint64(0x7FFFFFFF)  # a NaN's word, behind +inf

    def word(i):
        d = np.float32(((X[i] - q) ** 2).sum())
        return far if np.isnan(d) else np.uint64(d.view(np.uint32))

    pool = sorted([word(i), int(i), 1] for i in init)
    seen = set(int(i) for i in init)
    k = 0
    while k < len(pool):
        nk = len(pool)
        if pool[k][2]:
            pool[k][2] = 0
            for v in map(int, g[pool[k][1]]):
                if v in seen:
                    continue
                seen.add(v)
                w = word(v)
                if w >= pool[-1][0]:
                    continue
                at = sum(1 for e in pool if e[0] <= w)
                pool.insert(at, [w, v, 1])
                del pool[L:]
                nk = min(nk, at)
        k = nk if nk <= k else k + 1
    return pool


@pytest.mark.parametrize("L,bad", [(1, 1), (2, 1), (33, 1), (33, 5), (40, 40), (64, 0)])
@pytest.mark.parametrize("where", ["start", "start and neighbours", "query"])
def test_nan_rows(index, L, bad, where):
    n, d, W, m, k = 2000, 24, 20, 24, min(L, 10)
    rng = np.random.default_rng(3)
    X = rng.integers(-20, 21, (n, d)).astype(np.float32)
    X[:50, 5] = np.nan
    if where != "start":
        X[50::7, 2] = np.nan
    good = np.flatnonzero(~np.isnan(X).any(1))
    g = rng.choice(good if where == "start" else n, (n, W)).astype(np.uint32)
    init = np.stack([np.r_[np.arange(bad), rng.choice(good, L - bad, replace=False)] for _ in range(m)]).astype(np.uint32)
    Q = rng.integers(-20, 21, (m, d)).astype(np.float32)
    if where == "query":
        Q[::2, 0] = np.nan
    index.upload(X)
    index.set_graph(g, np.full(n, W, np.uint32), 0)
    gi, gd = index.search(Q, L, k, init)
    for i in range(m):
        pool = _one_by_one(X, g, Q[i], init[i], L)[:k]
        assert gi[i].tolist() == [e[1] for e in pool]
        want = np.array([e[0] for e in pool]).astype(np.uint32).view(np.float32)
        assert np.array_equal(gd[i], want, equal_nan=True)
