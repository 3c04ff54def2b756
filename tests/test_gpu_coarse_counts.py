"""The coarse step's statistics where every list is a near-tie: a query left to the
second pass counts its lists once, in the pass that scores them."""
import numpy as np
import pytest

import qann_b200 as qb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,redone", [(100, 0), (200, 200)])   # up to one query per SM the first pass holds every list
def test_each_list_counts_once(nq, redone):
    rng = np.random.default_rng(0)
    d, nlist = 32, 2048   # the first pass holds 1,024 candidates of 16 probes
    x = (rng.normal(size=d) + 1e-5 * rng.normal(size=(4 * nlist, d))).astype(np.float32)
    ivf = qb.IVFIndex(d, nlist, 16)
    ivf.enable_pq(16, fast_scan=True)
    ivf.train(x, max_iters=1, seed=1, clustering=qb.Clustering.Lloyd)
    ivf.add(x)
    q = x[rng.integers(0, len(x), nq)]
    qb.set_tensor_filter(2)
    try:
        before = qb.tensor_filter_counts()
        got = ivf.batch_query(q, 5)
        after = qb.tensor_filter_counts()
        qb.set_tensor_filter(0)
        want = ivf.batch_query(q, 5)
    finally:
        qb.set_tensor_filter(1)
    assert after["coarse_queries"] - before["coarse_queries"] == nq
    assert after["coarse_redone"] - before["coarse_redone"] == redone
    assert after["coarse_candidates"] - before["coarse_candidates"] == nq * nlist
    np.testing.assert_array_equal(got[0], want[0])
    assert got[1].tobytes() == want[1].tobytes()
