"""Exact k-NN through the sampled bound (bases above 40,960 rows, or many
queries): the FP32 filter, the tensor-core screen and the queries done again,
each equal to the oracle's brute force, ids and distances, ties by the lower id."""
import numpy as np
import pytest

from fastkcna_gb300 import synth

pytestmark = pytest.mark.gpu


def _rows(kind, n, d, seed):
    rng = np.random.default_rng(seed)
    if kind == "int":
        return np.ascontiguousarray(synth._draw("c2", n, seed)[:, :d])
    x = rng.standard_normal((n, d)).astype(np.float32)
    if kind == "offset":  # norms far above the distances: the screen passes too many rows
        x += np.float32(3000.0)
    elif kind == "large":
        x *= np.float32(1e17)
    elif kind == "tiny":
        x *= np.float32(1e-22)
    elif kind == "copies":  # 9,000 copies of one row
        x[5000:14000] = x[4]
    elif kind == "nan":
        x[::7, 0] = np.nan
    return x


@pytest.mark.parametrize("kind,n,d,m,k", [
    ("int", 45003, 128, 200, 100), ("normal", 45003, 128, 190, 1), ("normal", 66001, 61, 300, 500),
    ("normal", 300000, 32, 129, 10), ("offset", 45003, 128, 190, 10), ("large", 45003, 96, 260, 20),
    ("tiny", 45003, 96, 260, 20), ("normal", 41000, 200, 70, 33), ("int", 41000, 128, 3, 700),
    ("normal", 40961, 7, 1, 1), ("normal", 17001, 100, 2000, 12), ("normal", 40960, 20, 5, 64),
])
def test_bounded_knn_equals_brute_force(index, oracle, kind, n, d, m, k):
    X, Q = _rows(kind, n, d, 11), _rows(kind, m, d, 12)
    index.upload(X)
    gi, gd = index.knn_queries(Q, k)
    some = np.unique(np.r_[0, m - 1, np.arange(0, m, max(1, m // 40))])
    oi, od = oracle.knn_queries(X, Q[some], k)
    assert np.array_equal(gi[some], oi)
    assert np.array_equal(gd[some], od)


@pytest.mark.parametrize("kind,n,k", [
    ("normal", 300, 300), ("normal", 511, 256), ("normal", 512, 256), ("normal", 513, 257),
    ("normal", 4097, 256), ("normal", 20000, 10), ("nan", 4000, 256), ("levels", 3000, 256), ("levels", 9001, 7),
])
def test_small_base_selection(index, oracle, kind, n, k):
    """Selection from every distance: both sides of the thread minima's largest
    k, ragged rows per thread, and equal distances (six distinct ones, each held
    by fewer rows than a tie list, by more than the collected list together)."""
    d = 8
    X, Q = _rows("normal" if kind == "levels" else kind, n, d, 21), _rows("normal", 3, d, 22)
    if kind == "levels":
        X[:] = 0
        X[:, 0] = np.arange(n) % (6 if n < 6000 else 12)
        Q[:] = 0
    index.upload(X)
    gi, gd = index.knn_queries(Q, k)
    if kind == "nan":  # the oracle's insertion has no order for NaN; one more result takes the histogram passes
        oi, od = (a[:, :k] for a in index.knn_queries(Q, k + 1))
    else:
        oi, od = oracle.knn_queries(X, Q, k)
    assert np.array_equal(gi, oi) and np.array_equal(gd, od, equal_nan=True)


def test_bounded_knn_of_own_rows(index, oracle):
    X = _rows("int", 50001, 128, 13)
    index.upload(X)
    ids = np.arange(0, 50001, 250, dtype=np.uint32)
    gi, gd = index.knn_exact(ids, 50)
    oi, od = oracle.knn(X, ids[:40], 50)
    assert np.array_equal(gi[:40], oi) and np.array_equal(gd[:40], od)
    assert not (gi == ids[:, None]).any()


@pytest.mark.parametrize("kind", ["copies", "nan"])
def test_queries_done_again(index, kind):
    """More equal distances than a list holds, and NaN rows: the same answer as
    from a base small enough to be searched the first way."""
    X, Q = _rows(kind, 42000, 64, 17), _rows("normal", 500, 64, 18)
    index.upload(X)
    gi, gd = index.knn_queries(Q, 10)
    index.set_size(40960)
    si, sd = index.knn_queries(Q, 10)
    index.set_size(42000)
    inside = (gi < 40960).all(1)
    assert inside.sum() > 100
    assert np.array_equal(gi[inside], si[inside]) and np.array_equal(gd[inside], sd[inside])
