"""Exact k-NN at sizes where a bound pays (kcna_knn.cu, knn_bound_pays): the FP32
filter for few queries or long rows, the tensor-core screen for many, the
selection's two forms, rows that the screen cannot tell apart, and sizes next to
the lines; ids and distances equal to the oracle's brute force.  A call where it
does not pay is no slower than one with a few rows less, below the lines."""
import time

import numpy as np
import pytest

from fastkcna_gb300 import synth

pytestmark = pytest.mark.gpu


def _rows(kind, n, d, seed):
    rng = np.random.default_rng(seed)
    if kind == "int":
        return np.ascontiguousarray(synth._draw("c2", n, seed)[:, :d])
    x = rng.standard_normal((n, d), dtype=np.float32)
    if kind == "offset":  # norms far above the distances: the screen passes too many rows
        x += np.float32(3000.0)
    elif kind == "large":
        x *= np.float32(1e17)
    elif kind == "tiny":
        x *= np.float32(1e-22)
    elif kind == "nan":
        x[::7, 0] = np.nan
    return x


@pytest.mark.parametrize("kind,n,d,m,k", [
    # FP32 filter
    ("normal", 262143, 32, 3, 10), ("normal", 262144, 32, 3, 10), ("normal", 524288, 20, 9, 100),
    ("normal", 262147, 200, 70, 256), ("normal", 65536, 96, 2, 700), ("normal", 180001, 133, 33, 257),
    ("normal", 600011, 7, 1, 1), ("tiny", 262147, 100, 4, 20), ("large", 262147, 100, 4, 20),
    # screen
    ("int", 200003, 128, 400, 100), ("normal", 300000, 61, 500, 1), ("normal", 400003, 8, 1000, 300),
    ("normal", 1000003, 33, 129, 31), ("offset", 200003, 96, 400, 10), ("large", 200003, 96, 400, 20),
    ("tiny", 200003, 96, 400, 20),
])
def test_bounded_knn_equals_brute_force(index, oracle, kind, n, d, m, k):
    X, Q = _rows(kind, n, d, 11), _rows(kind, m, d, 12)
    index.upload(X)
    gi, gd = index.knn_queries(Q, k)
    some = np.unique(np.r_[0, m - 1, np.arange(0, m, max(1, m // 12))])
    oi, od = oracle.knn_queries(X, Q[some], k)
    assert np.array_equal(gi[some], oi)
    assert np.array_equal(gd[some], od)


@pytest.mark.parametrize("d,m", [(128, 400), (32, 4), (200, 20)])
def test_nan_rows(index, d, m):
    """A NaN row is farther than any other, whichever way finds the rows."""
    X, Q = _rows("nan", 300000, d, 17), _rows("normal", m, d, 18)
    index.upload(X)
    gi, gd = index.knn_queries(Q, 10)
    at = np.flatnonzero(~np.isnan(X[:, 0]))
    index.upload(X[at])
    si, sd = index.knn_queries(Q, 10)
    assert np.array_equal(gi, at[si]) and np.array_equal(gd, sd)


@pytest.mark.parametrize("n,below,d,m,k", [(41000, 40960, 960, 1, 10), (41000, 40960, 8, 256, 100), (65000, 16383, 8, 1000, 100)])
def test_no_step_up(index, n, below, d, m, k):
    rng = np.random.default_rng(5)
    X = rng.standard_normal((n, d), dtype=np.float32)
    Q = rng.standard_normal((m, d), dtype=np.float32)
    best = []
    for rows in (n, below):
        index.upload(X[:rows])
        index.knn_queries(Q, k)
        times = []
        for _ in range(41):
            t0 = time.perf_counter()
            index.knn_queries(Q, k)
            times.append(time.perf_counter() - t0)
        best.append(sorted(times)[5])
    assert best[0] < 1.25 * best[1] * n / below, best
