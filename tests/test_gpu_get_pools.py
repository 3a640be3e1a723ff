"""Pools read back in runs of nodes: a capacity that makes the last run short,
and outputs left out, against the pools that were set."""
import ctypes as C

import numpy as np
import pytest

from fastkcna_gb300 import kcna

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k", [(20011, 1000), (300, 7)])  # runs of 8,388 nodes; one run
def test_pools_read_back_as_set(index, n, k):
    rng = np.random.default_rng(k)
    X = rng.standard_normal((n, 4)).astype(np.float32)
    ids = ((np.arange(n)[:, None] + 1 + np.arange(k)) % n).astype(np.uint32)
    d = np.sort(rng.random((n, k)).astype(np.float32), axis=1)
    cnt = rng.integers(1, k + 1, n).astype(np.uint32)
    index.upload(X)
    index.set_pools(ids, d, cnt, kcna.params(K=k, L=k, S=10, search_L=min(k, 40), search_K=k))
    gi, gd, gc = index.pools()
    live = np.arange(gi.shape[1]) < cnt[:, None]
    assert np.array_equal(gc, cnt)
    assert np.array_equal(gi[live], ids[live[:, :k]]) and np.array_equal(gd[live], d[live[:, :k]])
    assert (gi[~live] == 0xFFFFFFFF).all() and np.isinf(gd[~live]).all()
    # into the middle of a buffer, ids only: nothing beside them is written
    buf = np.full(gi.size + 2, 7, np.uint32)
    rc = index.lib.kcna_get_pools(index.h, C.c_void_p(buf.ctypes.data + 4), None, None, C.c_uint32(gi.shape[1]))
    assert rc == 0 and buf[0] == 7 and buf[-1] == 7
    assert np.array_equal(buf[1:-1].reshape(gi.shape), gi)
