"""Contexts of several threads at once, with rows, beams and k of different
sizes: a kernel's shared-memory limit belongs to the whole process, so one
context's call must not narrow it for another's launch."""
import threading

import numpy as np
import pytest

from fastkcna_gb300 import kcna

pytestmark = pytest.mark.gpu


def _knn(ix, rng, d, size):
    ix.upload(rng.standard_normal((300000, d), dtype=np.float32))
    Q = rng.standard_normal((200, d)).astype(np.float32)
    return lambda: ix.knn_queries(Q, size)


def _search(ix, rng, d, size):
    n = 4000
    ix.upload(rng.standard_normal((n, d)).astype(np.float32))
    ix.set_graph(rng.integers(0, n, (n, 16)).astype(np.uint32), np.full(n, 16, np.uint32), 0)
    Q = rng.standard_normal((8, d)).astype(np.float32)
    init = np.stack([rng.choice(n, size, replace=False) for _ in range(8)]).astype(np.uint32)
    return lambda: ix.search(Q, size, 10, init)


def _rank_prune(ix, rng, d, size):
    n = 1500
    ix.upload(rng.standard_normal((n, d)).astype(np.float32))
    ids, dist = ix.knn_exact(np.arange(n, dtype=np.uint32), size)
    p = kcna.params(K=size, L=size, search_K=size, search_L=size)

    def run():
        ix.set_pools(ids, dist, np.full(n, size, np.uint32), p)
        ix.prune("cagra", p)
        return ix.graph()[:2]

    return run


def _build(ix, rng, d, size):
    ix.upload(rng.standard_normal((2500, d)).astype(np.float32))
    p = kcna.params(K=size, L=size, S=10, R=100, iterations=3, search_L=20, search_K=size, nsg_R=20, screen=1, tau=0.1)

    def run():  # no two builds of these are alike
        ix.build("taumng" if d >= 256 else "nsg", p)
        ids, dist, cnt = ix.pools()
        assert (cnt > 0).all() and (ids[:, 0] < 2500).all() and (np.diff(dist[:, :10]) >= 0).all()
        return ()

    return run


@pytest.mark.parametrize("make,forms", [(_build, [(24, 60), (300, 40), (64, 600), (130, 200)]), (_knn, [(128, 10), (96, 10), (200, 10)]), (_search, [(128, 1500), (1024, 1000), (32, 40)]),
                                        (_rank_prune, [(8, 1000), (8, 64), (8, 300)])])
def test_calls_of_several_threads(make, forms):
    errors = []
    start = threading.Barrier(len(forms))

    def job(d, size):
        try:
            with kcna.Index(0) as ix:
                run = make(ix, np.random.default_rng(d + size), d, size)
                start.wait(60)
                first = run()
                for _ in range(60):
                    assert all(np.array_equal(a, b) for a, b in zip(first, run()))
        except Exception as e:  # noqa: BLE001 (a thread's failure is the test's)
            errors.append(repr(e))
            start.abort()

    threads = [threading.Thread(target=job, args=f) for f in forms]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
