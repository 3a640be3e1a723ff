"""The FP32 warp prune with its batches in shared memory (rows of 32 to 192
floats) and without, against the oracle: both ends of that range, kept lists
that end in the first test's four rows, in one and in two chunks of 32 kept
rows and in the last few candidates of a batch, short pools, equal rows."""
import numpy as np
import oracle_py
import pytest

from fastkcna_gb300 import kcna

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", [1, 3, 4])
@pytest.mark.parametrize("d,k,R", [(28, 60, 32), (32, 33, 4), (61, 200, 5), (96, 260, 128), (189, 70, 36), (192, 100, 40),
                                   (193, 100, 37), (96, 2, 1)])
def test_warp_prune_equals_oracle(index, oracle, kind, d, k, R):
    n = 400
    rng = np.random.default_rng(d + k)
    X = rng.standard_normal((n, d)).astype(np.float32)
    X /= np.linalg.norm(X, axis=1, keepdims=True)
    X[50:90] = X[7]
    X[90:130] *= np.float32(0.25)
    index.upload(X)
    ids, dist = index.knn_exact(np.arange(n, dtype=np.uint32), k)
    cnt = np.full(n, k, np.uint32)
    cnt[::7] = 1
    cnt[3::7] = max(1, k // 3)
    kw = dict(K=k, L=k, S=10, R=100, iterations=1, search_L=40, nsg_R=R, search_K=k, tau=0.02, angle=60.0)
    kp = kcna.params(**kw)
    index.set_pools(ids, dist, cnt, kp)
    index.prune({1: "nsg", 3: "taumng", 4: "alphapg"}[kind], kp)
    g, deg, _ = index.graph()
    oi, _, odeg = oracle.prune(kind, X, oracle_py.params(**kw), ids, dist, cnt, g.shape[1])
    assert np.array_equal(deg, odeg)
    assert np.array_equal(g, oi)
