"""Calls on a device that others have nearly filled (KCNA_DEVICE_LIMIT_MB: an
allocation past the limit fails as cudaMalloc does): what ran in a given room
runs there still, with the same answers."""
import numpy as np
import pytest

from fastkcna_gb300 import kcna

pytestmark = pytest.mark.gpu


@pytest.fixture
def limited(monkeypatch):
    made = []

    def make(mb):
        monkeypatch.setenv("KCNA_DEVICE_LIMIT_MB", str(mb))
        ix = kcna.Index(0)
        monkeypatch.delenv("KCNA_DEVICE_LIMIT_MB")
        made.append(ix)
        return ix

    yield make
    for ix in made:
        ix.close()


# rows, queries and results take 48 MiB; every distance of 268 queries 1,022 MiB,
# the sampled ones of 1,088 and their lists 1,047
@pytest.mark.parametrize("mb", [1075, 1300])
def test_knn_within_a_limit(index, limited, mb):
    n, d, m, k = 1000000, 4, 2048, 1000
    rng = np.random.default_rng(2)
    X = rng.standard_normal((n, d)).astype(np.float32)
    Q = rng.standard_normal((m, d)).astype(np.float32)
    index.upload(X)
    want = index.knn_queries(Q, k)
    ix = limited(mb)
    ix.upload(X)
    for _ in range(2):
        got = ix.knn_queries(Q, k)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])


# rows 15 MiB, the graph and its copies about 100; bitmaps of four blocks an SM 290 MiB, of eight 580
@pytest.mark.parametrize("mb", [200, 480])
def test_search_within_a_limit(index, limited, mb):
    n, d, W, m, L = 1000000, 4, 8, 6000, 12
    rng = np.random.default_rng(3)
    X = rng.standard_normal((n, d)).astype(np.float32)
    g = rng.integers(0, n, (n, W)).astype(np.uint32)
    deg = np.full(n, W, np.uint32)
    Q = rng.standard_normal((m, d)).astype(np.float32)
    init = rng.integers(0, n, (m, L)).astype(np.uint32)
    out = []
    for ix in (index, limited(mb)):
        ix.upload(X)
        ix.set_graph(g, deg, 0)
        out.append(ix.search(Q, L, 5, init))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


# the pools take 45 MiB, the outputs taken apart 44 more
@pytest.mark.parametrize("mb", [50, 75, 400])
def test_pools_within_a_limit(limited, mb):
    n, cap = 60001, 97
    rng = np.random.default_rng(4)
    ids = rng.integers(0, n, (n, cap)).astype(np.uint32)
    dist = np.sort(rng.random((n, cap)).astype(np.float32), 1)
    cnt = rng.integers(0, cap + 1, n).astype(np.uint32)
    ix = limited(mb)
    ix.upload(rng.standard_normal((n, 4)).astype(np.float32))
    ix.set_pools(ids, dist, cnt, kcna.params(K=cap, L=cap, search_K=cap, search_L=cap))
    gi, gd, gc = ix.pools()
    assert np.array_equal(gc, cnt)
    there = np.arange(gi.shape[1])[None, :] < cnt[:, None]
    assert np.array_equal(gi, np.where(there, ids, np.uint32(0xFFFFFFFF)))
    assert np.array_equal(gd, np.where(there, dist, np.float32(np.inf)))
