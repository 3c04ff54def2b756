"""NaN scores come back as the one NaN that CUDA's arithmetic forms, from every kind of
index and by every path (an inner product is negated, and its key with it)."""
import numpy as np
import pytest

import qann_b200 as qb

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("kind", ["flat", "refine_flat", "refine"])
@pytest.mark.parametrize("k", [1, 10, 200])
def test_one_nan(kind, metric, k):
    rng = np.random.default_rng(0)
    x = rng.normal(size=(3000, 32)).astype(np.float32)
    q = rng.normal(size=(70, 32)).astype(np.float32)
    q[3, 5] = np.nan
    q[20, 0] = -np.nan
    q[69] = np.nan
    metric = qb.Metric(metric)
    if kind == "refine":
        idx = qb.IVFIndex(32, 100, 20, metric=metric)
        idx.enable_pq(16, fast_scan=True)
        idx.train(x, max_iters=1, seed=1, clustering=qb.Clustering.Lloyd)
    else:
        idx = qb.FlatIndex(32, metric=metric)
    if kind != "flat":
        idx = qb.RefineIndex(idx, 4)
    idx.add(x)
    try:
        for mode in (0, 1, 2):
            qb.set_tensor_filter(mode)
            for rows in (q, q[3:4]):
                ids, d = idx.batch_query(rows, k)
                nan = np.isnan(d)
                want = np.isnan(rows).any(1)[:, None] & (ids >= 0)
                np.testing.assert_array_equal(nan, want)
                assert (d[nan].view(np.uint32) == 0x7FFFFFFF).all()
    finally:
        qb.set_tensor_filter(1)
