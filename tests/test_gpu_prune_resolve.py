"""The FP8-screened prune hands nodes with undecided pairs to a second kernel,
in runs of at most 32,768 items: one item over a run, a range that stops the
scan inside a batch of pairs, and short pools, each against the FP32 prune of
the same pools (equal lists: the screen decides only what is certain)."""
import numpy as np
import pytest

from fastkcna_gb300 import kcna, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k,R", [(32769, 40, 12), (3001, 128, 128), (3001, 129, 1), (3001, 3, 50)])
def test_resolved_prune_identical_to_fp32(index, n, k, R):
    X = np.ascontiguousarray(synth.base("c4", n)[:, :257])
    index.upload(X)
    ids, d = index.knn_exact(np.arange(n, dtype=np.uint32), k)
    cnt = np.full(n, k, np.uint32)
    cnt[::5] = max(k // 2, 1)
    got = []
    for screen in (0, 1):
        p = kcna.params(K=k, L=k, search_K=k, search_L=min(k, 40), nsg_R=R, tau=1.0, screen=screen)
        index.set_pools(ids, d, cnt, p)
        index.prune("taumng", p)
        got.append(index.graph())
    assert np.array_equal(got[0][1], got[1][1])
    assert np.array_equal(got[0][0], got[1][0])
