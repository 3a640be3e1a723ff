"""P2K join of nodes whose new and old pushers together need more micro-tiles
than the lanes hold when each kind rounds up by itself (53 to 58 neighbours),
and of their neighbours in size: every pool distance after a refinement is the
distance of its pair (integer rows: exact in FP32), and no entry is listed twice."""
import numpy as np
import pytest

from fastkcna_gb300 import kcna

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pushes", [24, 40, 56])  # a round's pushes per node: units of 24 pushers, new and old mixed
@pytest.mark.parametrize("deg", [52, 53, 56, 58, 59, 70])
def test_p2k_distances_are_those_of_their_pairs(index, deg, pushes):
    n, d, L = 6000, 40, 64  # enough pushes for a warp's share to hold whole units
    rng = np.random.default_rng(deg)
    X = rng.integers(-40, 41, (n, d)).astype(np.float32)
    # pool and edges out of a node's 300 nearest: a round replaces a part of the pool, not all of it
    sq = (X.astype(np.float64) ** 2).sum(1)
    far = sq[:, None] + sq[None] - 2.0 * (X @ X.T)
    np.fill_diagonal(far, np.inf)
    near = np.argpartition(far, 300, axis=1)[:, :300]
    others = np.take_along_axis(near, rng.random((n, 300)).argsort(axis=1)[:, : L + deg], 1)

    def dists(ids):
        return ((X[ids].astype(np.int64) - X[:, None].astype(np.int64)) ** 2).sum(2)

    ids = others[:, :L].astype(np.uint32)
    dd = dists(ids)
    order = np.lexsort((ids, dd), axis=1)
    ids, dd = np.take_along_axis(ids, order, 1), np.take_along_axis(dd, order, 1).astype(np.float32)
    kp = kcna.params(K=L, L=L, S=10, R=100, iterations=1, search_L=L, nsg_R=50, search_K=L, massq_S=pushes, screen=0)
    index.upload(X)
    index.set_pools(ids, dd, np.full(n, L, np.uint32), kp)
    index.set_graph(others[:, L:].astype(np.uint32), np.full(n, deg, np.uint32), 0)
    assert index.refine(1, kp) > 0
    gi, gd, cnt = index.pools()
    assert (cnt == L).all()
    gi, gd = gi[:, :L], gd[:, :L]
    assert np.array_equal(gd, dists(gi).astype(np.float32))
    assert (np.diff(np.sort(gi, axis=1), axis=1) > 0).all()
    assert not np.array_equal(gi, ids)
