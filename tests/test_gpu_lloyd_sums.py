"""One Lloyd iteration from the starting rows (which leave no cluster empty: each is
nearest to itself), for L2 and for spherical k-means, at the widths the member
sums' kernels change at, against numpy: nearest in float64, members summed in
float32 one after the other, unit length by a float64 norm."""
import numpy as np
import pytest

import qann_b200 as qb

pytestmark = pytest.mark.gpu


def unit(x):
    s = np.zeros(len(x), np.float64)
    for c in range(x.shape[1]):
        v = x[:, c].astype(np.float64)
        s = s + v * v
    return x * (1.0 / np.sqrt(s)).astype(np.float32)[:, None]


def centroids(x, metric, iters):
    ivf = qb.IVFIndex(x.shape[1], 100, 8, metric=metric)
    ivf.train(x, max_iters=iters, seed=5, clustering=qb.Clustering.Lloyd)
    return ivf.centroids()


@pytest.mark.parametrize("spherical", [False, True])
@pytest.mark.parametrize("d", [1, 2, 3, 4, 5, 31, 32, 33, 65])
def test_one_iteration(d, spherical):
    if spherical and d == 1:
        pytest.skip("rows of one dimension are 1 or -1 at unit length: ties throughout")
    x = np.random.default_rng(40 + d).normal(size=(3000, d)).astype(np.float32)
    metric = qb.Metric.Cosine if spherical else qb.Metric.L2
    rows = unit(x) if spherical else x
    first, second = centroids(x, metric, 0), centroids(x, metric, 1)
    assert {r.tobytes() for r in first} <= {r.tobytes() for r in rows}   # the starting rows
    d2 = ((rows[:, None, :].astype(np.float64) - first[None].astype(np.float64)) ** 2).sum(2)
    label = d2.argmin(1)
    want = np.zeros_like(first)
    for c in range(len(first)):
        members = rows[label == c]
        assert len(members)
        s = np.zeros(d, np.float32)
        for r in members:
            s = s + r
        want[c] = s / np.float32(len(members))
    assert second.tobytes() == (unit(want) if spherical else want).tobytes()
