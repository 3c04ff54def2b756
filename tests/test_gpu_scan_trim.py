"""The scan's trims and its units' ends at the sizes where they can go wrong:
k' on either side of the buffers' multiples of 32, below and above the block
sort's bins, ties (equal sums, so equal distances) and constant distances,
against the reference-order oracle's semantics through the exact paths: every
scan shape and chunking must return the same bits."""
import numpy as np
import pytest

import qann_b200 as qb

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def defaults():
    yield
    qb.set_scan_options(autotune=True, variant=-1)


def index_of(kind, metric, n=12_000, d=32, m=16, nlist=120):
    rng = np.random.default_rng(11)
    x = rng.normal(size=(n, d)).astype(np.float32)
    if kind == "ties":       # few distinct rows: whole lists at one distance
        x = x[rng.integers(0, 40, n)]
    elif kind == "constant":
        x[:] = x[0]
        x += (1e-3 * rng.normal(size=(n, d)) * (rng.random((n, 1)) < 0.2)).astype(np.float32)
    ivf = qb.IVFIndex(d, nlist, 40, metric=qb.Metric(metric))
    ivf.enable_pq(m, fast_scan=True)
    ivf.train(x, max_iters=1, seed=2, clustering=qb.Clustering.Lloyd)
    ivf.add(x)
    return ivf, rng.normal(size=(9, d)).astype(np.float32)


@pytest.mark.parametrize("kind", ["normal", "ties", "constant"])
@pytest.mark.parametrize("metric", [0, 2])
@pytest.mark.parametrize("k", [1, 31, 32, 33, 64, 255, 257, 1000, 2048])
def test_shapes_agree(kind, metric, k):
    ivf, q = index_of(kind, metric)
    want = None
    for variant in (0, 1, 2):
        qb.set_scan_options(variant=variant, autotune=False)
        # alone a query is cut into chunks; 600 together are a unit each
        for batch in (q[:1], np.repeat(q, 67, axis=0)):
            ids, d = ivf.batch_query(batch, k)
            if want is None:
                want = ids[0], d[0]
            np.testing.assert_array_equal(ids[0], want[0])
            assert d[0].tobytes() == want[1].tobytes()


@pytest.mark.parametrize("kind", ["normal", "ties"])
def test_prefix_of_more(kind):
    """The k best are the first k of more: trims at different k' keep the same keys
    (with all of a query's vectors probed, ties by (distance, id) as sorted)."""
    ivf, q = index_of(kind, 0)
    ivf.nprobe = ivf.nlist
    big_ids, big_d = ivf.batch_query(q, 2000)
    for k in (1, 20, 100, 500):
        _, d = ivf.batch_query(q, k)
        assert d.tobytes() == np.ascontiguousarray(big_d[:, :k]).tobytes()
