"""The entry point is the row nearest the centroid: rows around one block of
1,024 and dimensions around one block of 64, in a beam over all but a few rows
(one row stands at the centroid of the others, far from any second)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(1024, 64), (1025, 65), (1039, 63), (1056, 129), (2071, 9)])
def test_entry_point_is_nearest_to_centroid(index, n, d):
    rng = np.random.default_rng(n + d)
    half = rng.integers(20, 120, ((n - 1) // 2, d)).astype(np.float32)
    X = np.zeros((n, d), np.float32)
    X[: len(half)] = half
    X[len(half): 2 * len(half)] = -half  # every sum is zero: rows left over stand at the origin
    order = rng.permutation(n)
    X = X[order]
    index.upload(X)
    index.build("nsg", K=40, L=40, S=8, R=60, iterations=4, search_L=40, nsg_R=16, search_K=40)
    _, _, ep = index.graph()
    assert not X[ep].any()
